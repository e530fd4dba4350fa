// tk_table.cu -- the k-mer count table: K2 count-insert, HLL sizing, rehash,
// K3 filter/histogram, sorted dump and the K4 ">COUNT\nKMER\n" formatter,
// and catalogue loading (a stored database or a jellyfish-style dump).
//
// Replaces `jellyfish count/histo/dump` as Trinity drives them
// (Trinity:2612-2638, util/insilico_read_normalization.pl:617-643).
//
// K2 walks the read array's 2-bit codes as one flat stream (thread_windows: 32
// window end positions a thread; a window is valid when no position in it is
// marked invalid, so read separators and N break k-mers with no per-read
// bookkeeping), buckets every window by its hash, and builds the table range
// by range in shared memory; a table that already holds keys is added to with
// atomics.  A key that finds no slot within max_probes goes to an overflow
// list; the host then doubles the table and re-inserts it, so no k-mer is ever
// dropped silently.
#include "tk_emit.cuh"
#include "tk_windows.cuh"

#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>

namespace tk {

constexpr int CT_THREADS = 256;
constexpr int CT_SPAN = 32;              // window end positions per thread
constexpr int HLL_P = 12;
constexpr int HLL_M = 1 << HLL_P;
constexpr int NBUCKETS = 1 << BUCKET_BITS;
constexpr int INS_PER_THREAD = 1;
// bucket passes: one 1024-thread block per SM (two threads to each 32 window
// end positions); each block stages up to SC_BUF keys per bucket in shared
// memory between flushes.  760M windows: 3.87 ms, with 512 threads 4.35.
constexpr int SC_THREADS = 1024;
constexpr int SC_TILE = 16384;                                   // window end positions per tile
// Positions of a set whose key buffer is not sized exactly: reading the size
// back is a round trip of about 12 us, 2% of the 600 us of one bin of 2000
// pairs and below 0.5% of the 3 ms that 2^24 positions take; the buffer is then
// at most a window at each position and three keys of padding per bucket and
// block, 138 MB with 152 blocks.
constexpr uint64_t SC_SMALL = 1ull << 24;
constexpr int SC_BUF = 24;                                       // a multiple of 4 (whole 32-byte sectors)
static_assert(SC_BUF % 4 == 0 && SC_BUF <= 32, "a half-warp flushes a bucket in two 16-key stores");
constexpr int SC_BUCKETS_PER_WARP = NBUCKETS / (SC_THREADS / 32);
static_assert((NBUCKETS / (SC_THREADS / 32)) % 2 == 0, "buckets are flushed in pairs");
constexpr size_t SC_SMEM = (size_t)NBUCKETS * SC_BUF * 8 + (size_t)NBUCKETS * 8 + (size_t)NBUCKETS * 4;
constexpr uint64_t INS_CHUNK = (uint64_t)CT_THREADS * INS_PER_THREAD;
enum NextMode { NEXT_NONE = 0, NEXT_FILL = 1, NEXT_PREFETCH = 2 };

// Pass 1a: k-mers per (hash bucket, column) and the HLL sketch of the batch.
// hist is bucket-major with `cols` columns per bucket; the read set uses the
// columns [col0, col0 + gridDim.x), one per block: hist[bucket * cols + col0 + block]
// (each read set has a histogram and key buffer of its own, col0 = 0).
// Each count is rounded up to a multiple of 4 keys, so every (bucket, column)
// region of the key buffer starts on a 32-byte sector; pass 1b pads the
// rounding with EMPTY_KEY, which the insert skips.  Pass 1b's block owns tiles
// b, b+G, b+2G, ... (G blocks); this pass covers the same tiles, two at a time.
constexpr int HIST_THREADS = 1024;
template <bool CANON>
__global__ void __launch_bounds__(HIST_THREADS) k_part_hist(const uint64_t *__restrict__ codes,
                                                           const uint32_t *__restrict__ inv, uint64_t n, int k,
                                                           uint32_t *__restrict__ hist, uint64_t cols, uint64_t col0,
                                                           uint32_t *__restrict__ regs,
                                                           unsigned long long *__restrict__ windows_out) {
    __shared__ uint32_t sh[NBUCKETS];
    __shared__ uint32_t sreg[HLL_M];
    for (int i = threadIdx.x; i < NBUCKETS; i += HIST_THREADS) sh[i] = 0;
    for (int i = threadIdx.x; i < HLL_M; i += HIST_THREADS) sreg[i] = 0;
    __syncthreads();
    uint32_t windows = 0;
    const uint64_t tile = SC_TILE;
    const uint32_t half = threadIdx.x / (SC_TILE / CT_SPAN), t = threadIdx.x % (SC_TILE / CT_SPAN);
    for (uint64_t base = ((uint64_t)blockIdx.x + (uint64_t)half * gridDim.x) * tile; base < n;
         base += 2ull * gridDim.x * tile) {
        const uint64_t p0 = base + (uint64_t)t * CT_SPAN;
        thread_windows<CANON>(codes, inv, p0 >> 5, p0 < n, k, [&](uint64_t key, int) {
            uint64_t h = mix64(key);
            atomicAdd(&sh[h >> (64 - BUCKET_BITS)], 1u);
            uint32_t idx = (uint32_t)(h & (HLL_M - 1));
            uint32_t rank = (uint32_t)__clzll((long long)(h >> HLL_P)) - HLL_P + 1u;
            if (rank > sreg[idx]) atomicMax(&sreg[idx], rank);
            windows++;
        });
    }
    __syncthreads();
    for (int i = threadIdx.x; i < NBUCKETS; i += HIST_THREADS) hist[(uint64_t)i * cols + col0 + blockIdx.x] = (sh[i] + 3u) & ~3u;
    for (int i = threadIdx.x; i < HLL_M; i += HIST_THREADS)
        if (sreg[i]) atomicMax(&regs[i], sreg[i]);
    windows = warp_sum(windows);
    if (lane_id() == 0 && windows) atomicAdd(windows_out, (unsigned long long)windows);
}

// Pass 1b: the same windows (same grid, same tiles as pass 1a), written
// bucket-major into the key buffer.  A random 8-byte store leaves its 32-byte
// sector partly written, and L2 then reads the sector from DRAM before it can
// write it back; so the keys of a tile are staged per bucket in shared memory
// and leave the block as whole, aligned sectors.  Per bucket the block keeps
// gpos (where its next staged key goes; a multiple of 4 keys) and cnt (keys
// staged, including up to 3 carried over from the previous tile).  A key
// ranked past SC_BUF in one tile (a bucket flooded by a repeat) is stored
// directly at its final position.  After each tile the warp that owns a
// bucket writes its whole sectors and moves the 0-3 key remainder to the
// front; at the end the remainders go out padded with EMPTY_KEY.
template <bool CANON>
__global__ void __launch_bounds__(SC_THREADS, 1) k_part_scatter(const uint64_t *__restrict__ codes,
                                                               const uint32_t *__restrict__ inv, uint64_t n, int k,
                                                               const uint64_t *__restrict__ offs, uint64_t cols,
                                                               uint64_t col0, uint64_t *__restrict__ keys,
                                                               const uint32_t *__restrict__ wait_err) {
    if (*wait_err) return;   // the offsets' scan gave up: they are not to be stored by
    extern __shared__ __align__(16) unsigned char sc_smem[];
    uint64_t *buf = reinterpret_cast<uint64_t *>(sc_smem);                       // [NBUCKETS][SC_BUF]
    unsigned long long *gpos = reinterpret_cast<unsigned long long *>(buf + (size_t)NBUCKETS * SC_BUF);
    uint32_t *cnt = reinterpret_cast<uint32_t *>(gpos + NBUCKETS);
    for (int i = threadIdx.x; i < NBUCKETS; i += SC_THREADS) {
        gpos[i] = offs[(uint64_t)i * cols + col0 + blockIdx.x];
        cnt[i] = 0;
    }
    __syncthreads();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint64_t stride = (uint64_t)gridDim.x * SC_TILE;
    for (uint64_t base = (uint64_t)blockIdx.x * SC_TILE; base < n; base += stride) {
        const uint64_t p0 = base + (uint64_t)(threadIdx.x % (SC_TILE / CT_SPAN)) * CT_SPAN;
        auto put = [&](uint64_t key, int) {
            const uint32_t b = (uint32_t)(mix64(key) >> (64 - BUCKET_BITS));
            const uint32_t r = atomicAdd(&cnt[b], 1u);
            if (r < SC_BUF) buf[b * SC_BUF + r] = key;
            else keys[gpos[b] + r] = key;
        };
        static_assert(SC_THREADS == 2 * (SC_TILE / CT_SPAN), "two threads per 32 positions");
        if (threadIdx.x < SC_TILE / CT_SPAN) thread_windows<CANON, 0, 16>(codes, inv, p0 >> 5, p0 < n, k, put);
        else thread_windows<CANON, 16, 32>(codes, inv, p0 >> 5, p0 < n, k, put);
        __syncthreads();
        // two buckets per step, one per half-warp
        const unsigned hl = lane & 15u;
        for (int i = 0; i < SC_BUCKETS_PER_WARP; i += 2) {
            const int b = warp * SC_BUCKETS_PER_WARP + i + (int)(lane >> 4);
            const uint32_t nk = cnt[b];
            const uint32_t full = nk & ~3u;
            const uint64_t g = gpos[b];
            const uint64_t *bb = buf + (size_t)b * SC_BUF;
            const uint32_t nb = min(full, (uint32_t)SC_BUF);
            if (hl < nb) keys[g + hl] = bb[hl];
            if (hl + 16 < nb) keys[g + hl + 16] = bb[hl + 16];
            const uint32_t tail = nk - full;
            uint64_t v = 0;
            if (hl < tail) {
                const uint32_t idx = full + hl;
                v = idx < SC_BUF ? bb[idx] : __ldcg(keys + g + idx);
            }
            __syncwarp();
            if (hl < tail) buf[(size_t)b * SC_BUF + hl] = v;
            if (hl == 0) {
                cnt[b] = tail;
                gpos[b] = g + full;
            }
            __syncwarp();
        }
        __syncthreads();
    }
    for (int i = 0; i < SC_BUCKETS_PER_WARP; i++) {
        const int b = warp * SC_BUCKETS_PER_WARP + i;
        const uint32_t nk = cnt[b];
        if (nk && lane < 4) keys[gpos[b] + lane] = lane < nk ? buf[(size_t)b * SC_BUF + lane] : EMPTY_KEY;
    }
}

__device__ __forceinline__ void l2_prefetch_bulk(const void *p, uint32_t bytes) {
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"(bytes) : "memory");
}

// Pass 2, per partition p: a launch that prepares slice p (fill >= 0, p = -1)
// -- on a fresh table it writes the empty slots (those writes allocate in L2,
// so the slice is never read from DRAM); on a table that already holds keys it
// bulk-prefetches the slice to L2 -- then a launch that inserts partition p's
// keys (fill = -1).  Stream order between the launches is the only
// synchronisation.
__global__ void __launch_bounds__(CT_THREADS) k_part_step(const uint64_t *__restrict__ keys,
                                                         const uint64_t *__restrict__ offs, uint64_t cols, int p,
                                                         int fill, DevTable t, int next_mode, int max_probes,
                                                         uint64_t *__restrict__ ovf_keys, uint32_t *__restrict__ ovf_cnt,
                                                         uint64_t ovf_cap, unsigned long long *__restrict__ counters) {
    const int nparts = 1 << t.pbits;
    const uint64_t nslot = t.lmask + 1;
    if (fill >= 0 && fill < nparts) {
        Slot *nxt = t.slots + ((uint64_t)fill << t.lbits);
        if (next_mode == NEXT_FILL) {
            ulonglong2 e;
            e.x = EMPTY_KEY;
            e.y = 0;
            ulonglong2 *v = reinterpret_cast<ulonglong2 *>(nxt);
            for (uint64_t i = (uint64_t)blockIdx.x * CT_THREADS + threadIdx.x; i < nslot; i += (uint64_t)gridDim.x * CT_THREADS)
                v[i] = e;
        } else if (next_mode == NEXT_PREFETCH && threadIdx.x == 0) {
            const uint64_t bytes = nslot * sizeof(Slot);
            const uint64_t share = ((bytes + gridDim.x - 1) / gridDim.x + 15) & ~15ULL;
            uint64_t lo = (uint64_t)blockIdx.x * share;
            const uint64_t hi = min(bytes, lo + share);
            const char *base = reinterpret_cast<const char *>(nxt);
            for (int q = 0; q < 8 && lo < hi; q++) {   // 16-byte aligned start, multiple-of-16 size, <= 64 KB each
                uint64_t b = min(hi - lo, (uint64_t)65536);
                l2_prefetch_bulk(base + lo, (uint32_t)b);
                lo += b;
            }
        }
    }
    if (p < 0) return;
    const uint64_t bpp = (uint64_t)(NBUCKETS >> t.pbits);
    const uint64_t ps = offs[(uint64_t)p * bpp * cols];
    const uint64_t pe = offs[(uint64_t)(p + 1) * bpp * cols];
    for (uint64_t base = ps + (uint64_t)blockIdx.x * INS_CHUNK; base < pe; base += (uint64_t)gridDim.x * INS_CHUNK) {
        uint64_t kk[INS_PER_THREAD], s[INS_PER_THREAD];
        unsigned long long cur[INS_PER_THREAD];
#pragma unroll
        for (int j = 0; j < INS_PER_THREAD; j++) {
            uint64_t i = base + (uint64_t)j * CT_THREADS + threadIdx.x;
            kk[j] = i < pe ? __ldcs(keys + i) : EMPTY_KEY;
            s[j] = tbl_home(t, mix64(kk[j]));
        }
        // first probes of all keys issued back to back
#pragma unroll
        for (int j = 0; j < INS_PER_THREAD; j++) cur[j] = kk[j] != EMPTY_KEY ? tbl_claim(&t.slots[s[j]], kk[j]) : 0ULL;
#pragma unroll
        for (int j = 0; j < INS_PER_THREAD; j++) {
            if (kk[j] == EMPTY_KEY) continue;
            const uint64_t key = kk[j];
            uint64_t slot = s[j];
            unsigned long long c = cur[j];
            bool done = false;
            for (int probe = 0; probe < max_probes; probe++) {
                if (probe) c = tbl_claim(&t.slots[slot], key);
                if (c == key) {
                    atomicAdd(&t.slots[slot].val, 1u);
                    done = true;
                    break;
                }
                slot = tbl_next(t, slot);
            }
            if (!done) {
                unsigned long long o = atomicAdd(&counters[0], 1ULL);
                if (o < ovf_cap) { ovf_keys[o] = key; ovf_cnt[o] = 1u; }
            }
        }
    }
}

// ---- pass 2 by ranges (slices of at least 2^SR_MIN_LBITS slots), a batch of
// partitions at a time.  k_sr_group cuts each partition's keys into chunks and
// sorts every chunk by the range of the slice its keys' home slots fall in (a
// slice is cut into SR_BUILD_PER_SM ranges per SM); a chunk needs nothing from
// the others, so the keys are read once and no totals are known beforehand.
// k_sr_build then takes a block per range: it gathers the range's run of every
// chunk, builds the range in shared memory (all empty at first) with
// shared-memory CAS and add, and writes the range back whole.  A key whose
// probe run reaches the end of its range (its chain goes on into the next
// range, which another block owns) is merged into a small per-block table and
// then appended with its multiplicity to a deferred list that is inserted into
// the global table once every range is written; the global probe order (home,
// home+1, ... wrapping in the slice) is the one every reader uses, so the
// layout is an ordinary linear-probing table.  Global atomics drop from two
// per occurrence to the deferred keys alone, and a fresh slice needs no
// separate fill.
//
// A batch holds about SR_BATCH_KEYS keys (256 MB of grouped keys): what counts
// is that a launch has many blocks, whose loads, inserts and writes overlap, not
// that the grouped keys are still in L2 when the build reads them.  5M pairs
// (760M keys, 256 partitions), group + build: 6M keys a batch 3.9 + 8.0 ms, 12M
// 3.4 + 6.1, 24M 3.2 + 5.7, 48M 3.1 + 5.5, 96M 3.1 + 5.4 (the histogram,
// regrouping and build of one partition after another that this replaces: 2.7 +
// 5.4 + 6.8).  The group is bound by memory and its shared-memory sort (3.9
// TB/s), the build by its probes' instructions (180 per 32 keys).  Ranges of
// half the size with 512-thread blocks 6.3, of twice the size 6.9, 768-thread
// blocks 6.0 ms at 48M; chunks of 4096 (three blocks per SM) and 8192 keys
// (one) 3.2 and 4.8.
constexpr int SR_MIN_LBITS = 12;        // slices below 4096 slots keep the atomic path
constexpr int SR_BUILD_PER_SM = 2;      // ranges per slice and SM
constexpr int SR_MAX_SLOTS = 7168;      // slots of one range in shared memory (12 bytes each)
constexpr int SR_BUILD_THREADS = 1024;
constexpr int SR_MINI = 64;
constexpr int SG_THREADS = 512;
constexpr int SG_KEYS = 12;             // keys per thread, in registers
constexpr uint32_t SG_CHUNK = SG_THREADS * SG_KEYS;
constexpr uint64_t SR_BATCH_KEYS = 32ull << 20;

// A slice of 2^lbits slots is cut into nsub ranges: slot s belongs to range
// floor(s * nsub / 2^lbits), so range r is [ceil(r 2^lbits / nsub),
// ceil((r+1) 2^lbits / nsub)).
__device__ __forceinline__ uint32_t slot_range(const DevTable &t, uint64_t s, uint32_t nsub) {
    return (uint32_t)((s * nsub) >> t.lbits);
}
__device__ __forceinline__ uint64_t range_first(const DevTable &t, uint32_t r, uint32_t nsub) {
    return (((uint64_t)r << t.lbits) + nsub - 1) / nsub;
}
__device__ __forceinline__ uint32_t key_range(const DevTable &t, uint64_t key, uint32_t nsub) {
    return slot_range(t, mix64(key) & t.lmask, nsub);
}

// A partition's keys: one segment of each read set's bucket buffer, taken
// as one sequence (index i of segment s is key cum[s] + i of the sequence).
struct KeySeg {
    const uint64_t *keys;
    uint64_t len;
};
constexpr int MAX_KEY_SEGS = (int)COUNT_MAX_SETS;   // read sets counted in one pass (more are counted in groups)

struct SegView {
    const uint64_t *ptr[MAX_KEY_SEGS];
    uint64_t cum[MAX_KEY_SEGS + 1];
    uint32_t n;
};

// Loads the partition's segment table into shared memory (all threads).
__device__ __forceinline__ void seg_view_load(SegView &v, const KeySeg *__restrict__ segs, uint32_t nseg) {
    if (threadIdx.x == 0) {
        uint64_t c = 0;
        for (uint32_t s = 0; s < nseg; s++) {
            v.ptr[s] = segs[s].keys;
            v.cum[s] = c;
            c += segs[s].len;
        }
        v.cum[nseg] = c;
        v.n = nseg;
    }
    __syncthreads();
}

// A thread's walk over ascending sequence indices: the current segment's
// pointer, first index and end in registers; shared memory is read only when
// the walk crosses into a later segment.
struct SegCursor {
    const uint64_t *ptr;
    uint64_t first, end;
    uint32_t s;
};

__device__ __forceinline__ void seg_cursor_at(const SegView &v, SegCursor &c, uint32_t s) {
    c.s = s;
    c.ptr = v.ptr[s];
    c.first = v.cum[s];
    c.end = v.cum[s + 1];
}

// Key i of the sequence (i at or after every index the cursor gave before).
__device__ __forceinline__ uint64_t seg_key(const SegView &v, SegCursor &c, uint64_t i) {
    while (i >= c.end && c.s + 1 < v.n) seg_cursor_at(v, c, c.s + 1);
    return __ldcs(c.ptr + (i - c.first));
}

// The segment holding sequence index i.
__device__ __forceinline__ uint32_t seg_of(const SegView &v, uint64_t i) {
    uint32_t s = 0;
    while (s + 1 < v.n && i >= v.cum[s + 1]) s++;
    return s;
}

// A partition's chunks in its batch's buffers.
struct PartGeom {
    uint32_t chunk0, chunks;
};

// Chunk blockIdx.x of the batch, sorted by range into out[blockIdx.x *
// SG_CHUNK ...]; starts[blockIdx.x * (nsub + 1) + r] = where range r's run
// begins (entry nsub: the chunk's keys without the EMPTY_KEY padding).
__global__ void __launch_bounds__(SG_THREADS, 2) k_sr_group(const KeySeg *__restrict__ segs, uint32_t nseg,
                                                           const PartGeom *__restrict__ parts, uint32_t n_parts,
                                                           DevTable t, uint32_t nsub, uint64_t *__restrict__ out,
                                                           uint16_t *__restrict__ starts) {
    extern __shared__ __align__(16) unsigned char sg_smem[];
    uint64_t *skeys = reinterpret_cast<uint64_t *>(sg_smem);               // [SG_CHUNK]
    uint32_t *cnt = reinterpret_cast<uint32_t *>(skeys + SG_CHUNK);        // [nsub]
    __shared__ uint32_t sm[SG_THREADS / 32 + 1];
    __shared__ SegView sv;
    uint32_t lo = 0, hi = n_parts;   // the chunk's partition (partitions without chunks share a first one)
    while (hi - lo > 1) {
        const uint32_t mid = (lo + hi) >> 1;
        if (parts[mid].chunk0 <= blockIdx.x) lo = mid; else hi = mid;
    }
    for (uint32_t r = threadIdx.x; r < nsub; r += SG_THREADS) cnt[r] = 0;
    seg_view_load(sv, segs + (uint64_t)lo * nseg, nseg);   // synchronises
    const uint64_t n = sv.cum[sv.n], c0 = (uint64_t)(blockIdx.x - parts[lo].chunk0) * SG_CHUNK;
    SegCursor cur;
    seg_cursor_at(sv, cur, seg_of(sv, c0));
    uint64_t key[SG_KEYS];
    uint32_t at[SG_KEYS];   // (range << 16) | rank in the chunk's run of it
#pragma unroll
    for (int u = 0; u < SG_KEYS; u++) {
        const uint64_t i = c0 + (uint64_t)u * SG_THREADS + threadIdx.x;   // ascending over u
        key[u] = i < n ? seg_key(sv, cur, i) : EMPTY_KEY;
    }
#pragma unroll
    for (int u = 0; u < SG_KEYS; u++) {
        at[u] = 0;
        if (key[u] != EMPTY_KEY) {
            const uint32_t r = key_range(t, key[u], nsub);
            at[u] = r << 16 | atomicAdd(&cnt[r], 1u);
        }
    }
    __syncthreads();
    // counts -> starts (thread t sums a run of consecutive ranges)
    const uint32_t per = (nsub + SG_THREADS - 1) / SG_THREADS;
    const uint32_t r0 = min(nsub, threadIdx.x * per), r1 = min(nsub, r0 + per);
    uint32_t sum = 0, m;
    for (uint32_t r = r0; r < r1; r++) sum += cnt[r];
    uint32_t run = block_excl_scan<uint32_t>(sum, sm, &m);
    uint16_t *st = starts + (uint64_t)blockIdx.x * (nsub + 1);
    for (uint32_t r = r0; r < r1; r++) {
        const uint32_t c = cnt[r];
        cnt[r] = run;
        st[r] = (uint16_t)run;
        run += c;
    }
    if (threadIdx.x == 0) st[nsub] = (uint16_t)m;
    __syncthreads();
#pragma unroll
    for (int u = 0; u < SG_KEYS; u++)
        if (key[u] != EMPTY_KEY) skeys[cnt[at[u] >> 16] + (at[u] & 0xFFFFu)] = key[u];
    __syncthreads();
    uint64_t *o = out + (uint64_t)blockIdx.x * SG_CHUNK;
    for (uint32_t i = 2 * threadIdx.x; i < m; i += 2 * SG_THREADS)   // SG_CHUNK is even: the last pair stays inside
        *reinterpret_cast<ulonglong2 *>(o + i) = *reinterpret_cast<const ulonglong2 *>(skeys + i);
}

// Shared-memory probe from `loc` up to `end` in a table kept as separate key
// and count arrays (8-byte keys: a warp's random probes hit half as many banks
// per slot as 16-byte slots would); adds `inc` where the key lives or lands.
// A slot's key never changes once set, so a plain load that sees the key (most
// occurrences repeat a key already placed) needs only the add; an empty slot
// is claimed with CAS (counted in `added`).  A step looks at an aligned pair of
// slots (one 16-byte load; 6% of the build).  `keys` has an even number of
// entries.  Returns false if the probe ran off the end.
__device__ __forceinline__ bool smem_add(unsigned long long *keys, uint32_t *vals, uint32_t loc, uint32_t end,
                                         uint64_t key, uint32_t inc, uint32_t &added) {
    while (loc < end) {
        unsigned long long a, b;
        asm volatile("ld.volatile.shared.v2.u64 {%0, %1}, [%2];"
                     : "=l"(a), "=l"(b)
                     : "r"((uint32_t)__cvta_generic_to_shared(&keys[loc & ~1u])));
        unsigned long long cur = loc & 1u ? b : a;
        if (!(loc & 1u) && cur != key && cur != EMPTY_KEY) {
            cur = b;
            if (++loc >= end) return false;
        }
        if (cur == EMPTY_KEY) cur = atomicCAS(&keys[loc], EMPTY_KEY, (unsigned long long)key);
        if (cur == EMPTY_KEY || cur == key) {
            added += cur == EMPTY_KEY;
            atomicAdd(&vals[loc], inc);
            return true;
        }
        loc++;
    }
    return false;
}

struct __align__(16) BuildSmem {
    unsigned long long tkey[SR_MAX_SLOTS], mkey[SR_MINI];   // 16-byte aligned pairs
    uint32_t tval[SR_MAX_SLOTS], mval[SR_MINI];
    uint64_t run[SR_BUILD_THREADS];          // where the chunk's run begins in the grouped keys, less cum (64-bit: a
                                             // partition of deep reads over few k-mers may be more than 2^32 keys)
    uint32_t cum[SR_BUILD_THREADS + 1];      // keys of the range in the chunks before
    uint32_t scan[SR_BUILD_THREADS / 32 + 1];
};

// Range blockIdx.x % nsub of partition p0 + blockIdx.x / nsub.
__global__ void __launch_bounds__(SR_BUILD_THREADS) k_sr_build(const uint64_t *__restrict__ grouped,
                                                        const uint16_t *__restrict__ starts,
                                                        const PartGeom *__restrict__ parts, uint32_t nsub, int p0,
                                                        DevTable t, uint64_t *__restrict__ defer_keys,
                                                        uint32_t *__restrict__ defer_cnt, uint64_t defer_cap,
                                                        unsigned long long *__restrict__ defer_n,
                                                        unsigned long long *__restrict__ distinct) {
    extern __shared__ __align__(16) unsigned char sr_smem[];
    BuildSmem &sm = *reinterpret_cast<BuildSmem *>(sr_smem);
    const uint32_t pb = blockIdx.x / nsub, r = blockIdx.x % nsub;
    const PartGeom part = parts[pb];
    const uint64_t r0 = range_first(t, r, nsub);
    const uint32_t len = (uint32_t)(range_first(t, r + 1, nsub) - r0);   // <= SR_MAX_SLOTS (host checks)
    for (uint32_t i = threadIdx.x; i < len; i += SR_BUILD_THREADS) {
        sm.tkey[i] = EMPTY_KEY;
        sm.tval[i] = 0;
    }
    for (int i = threadIdx.x; i < SR_MINI; i += SR_BUILD_THREADS) {
        sm.mkey[i] = EMPTY_KEY;
        sm.mval[i] = 0;
    }
    const unsigned lane = lane_id(), warp = threadIdx.x >> 5;
    uint32_t added = 0, unused = 0;
    for (uint32_t t0 = 0; t0 < part.chunks; t0 += SR_BUILD_THREADS) {
        // the runs of up to SR_BUILD_THREADS chunks, taken as one sequence
        const uint32_t c = t0 + threadIdx.x;
        uint32_t n = 0;
        uint64_t first = 0;
        if (c < part.chunks) {
            const uint16_t *st = starts + (uint64_t)(part.chunk0 + c) * (nsub + 1) + r;
            const uint32_t a = st[0];
            n = st[1] - a;
            first = (uint64_t)(part.chunk0 + c) * SG_CHUNK + a;
        }
        uint32_t total;
        const uint32_t before = block_excl_scan<uint32_t>(n, sm.scan, &total);
        sm.cum[threadIdx.x] = before;
        sm.run[threadIdx.x] = first - before;
        if (threadIdx.x == 0) sm.cum[SR_BUILD_THREADS] = total;
        __syncthreads();
        // a warp takes a stretch of the sequence; a lane walks its runs forward
        const uint32_t per = (total + SR_BUILD_THREADS - 1) / SR_BUILD_THREADS * 32;
        const uint32_t lo = warp * per, hi = min(total, lo + per);
        uint32_t q = 0;
        if (lo < hi) {
            uint32_t e = SR_BUILD_THREADS;   // cum[q] <= lo < cum[e]
            while (e - q > 1) {
                const uint32_t mid = (q + e) >> 1;
                if (sm.cum[mid] <= lo) q = mid; else e = mid;
            }
        }
        auto put = [&](uint64_t key, uint32_t inc) {
            if (smem_add(sm.tkey, sm.tval, (uint32_t)((mix64(key) & t.lmask) - r0), len, key, inc, added)) return;
            // the probe left the range: count it in the per-block table, or defer it
            const uint32_t m = (uint32_t)(mix64(key ^ 0x5851F42D4C957F2DULL) & (SR_MINI - 1));
            if (smem_add(sm.mkey, sm.mval, m, SR_MINI, key, inc, unused) ||
                (m && smem_add(sm.mkey, sm.mval, 0, m, key, inc, unused)))
                return;
            const unsigned long long j = atomicAdd(defer_n, 1ULL);
            if (j < defer_cap) {
                defer_keys[j] = key;
                defer_cnt[j] = inc;
            }
        };
        for (uint32_t i0 = lo + lane; i0 - lane < hi; i0 += 128) {
            uint64_t k4[4];
#pragma unroll
            for (int u = 0; u < 4; u++) {
                const uint32_t i = i0 + u * 32;
                k4[u] = EMPTY_KEY;
                if (i < hi) {
                    while (sm.cum[q + 1] <= i) q++;
                    k4[u] = __ldcg(grouped + (sm.run[q] + i));
                }
            }
            // A repeat's key: one add for the warp's 128 (without it the one block
            // that holds poly-A is what the call waits for: 400,000 reads, half of them
            // poly-A, 7.5 ms for 4.5).  The loop is uniform over the warp, and the vote
            // brings its lanes together before the probes: 3M reads of a 40 Mb genome
            // 2.83 -> 2.69 ms, of 20 kb over and over 5.7 -> 4.0.
            const uint64_t k0 = __shfl_sync(0xffffffffu, k4[0], 0);   // (every lane takes it)
            const bool alike = (k4[0] == k0) & (k4[1] == k0) & (k4[2] == k0) & (k4[3] == k0);
            if (__all_sync(0xffffffffu, alike)) {
                if (lane == 0 && k0 != EMPTY_KEY) put(k0, 128u);
                continue;
            }
#pragma unroll
            for (int u = 0; u < 4; u++)
                if (k4[u] != EMPTY_KEY) put(k4[u], 1u);
        }
        __syncthreads();
    }
    __syncthreads();
    added = warp_sum(added);
    if (lane == 0 && added) atomicAdd(distinct, (unsigned long long)added);
    ulonglong2 *g = reinterpret_cast<ulonglong2 *>(t.slots + ((uint64_t)(p0 + pb) << t.lbits) + r0);
    for (uint32_t i = threadIdx.x; i < len; i += SR_BUILD_THREADS) {
        ulonglong2 v;
        v.x = sm.tkey[i];
        v.y = sm.tval[i];
        g[i] = v;
    }
    for (int i = threadIdx.x; i < SR_MINI; i += SR_BUILD_THREADS) {
        if (sm.mkey[i] == EMPTY_KEY) continue;
        const unsigned long long j = atomicAdd(defer_n, 1ULL);
        if (j < defer_cap) {
            defer_keys[j] = sm.mkey[i];
            defer_cnt[j] = sm.mval[i];
        }
    }
}

__global__ void k_rehash(const Slot *__restrict__ old, uint64_t old_cap, DevTable t, int max_probes,
                         uint64_t *__restrict__ ovf_keys, uint32_t *__restrict__ ovf_cnt, uint64_t ovf_cap,
                         unsigned long long *__restrict__ counters) {
    uint32_t added = 0;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < old_cap; i += (uint64_t)gridDim.x * blockDim.x) {
        ulonglong2 v = __ldcs(reinterpret_cast<const ulonglong2 *>(&old[i]));
        if (v.x == EMPTY_KEY) continue;
        if (!tbl_add_new(t, v.x, (uint32_t)v.y, max_probes, &added)) {
            unsigned long long j = atomicAdd(&counters[0], 1ULL);
            if (j < ovf_cap) { ovf_keys[j] = v.x; ovf_cnt[j] = (uint32_t)v.y; }
        }
    }
}

__global__ void k_insert_pairs(const uint64_t *__restrict__ keys, const uint32_t *__restrict__ cnt, uint64_t n, DevTable t,
                               int max_probes, uint64_t *__restrict__ ovf_keys, uint32_t *__restrict__ ovf_cnt,
                               uint64_t ovf_cap, unsigned long long *__restrict__ counters) {
    uint32_t added = 0;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        uint64_t key = keys[i];
        uint32_t c = cnt ? cnt[i] : 1u;
        if (!tbl_add_new(t, key, c, max_probes, &added)) {
            unsigned long long j = atomicAdd(&counters[0], 1ULL);
            if (j < ovf_cap) { ovf_keys[j] = key; ovf_cnt[j] = c; }
        }
    }
}

// The deferred keys of a range build (*n of them; none when they overran cap).
__global__ void k_insert_deferred(const uint64_t *__restrict__ keys, const uint32_t *__restrict__ cnt,
                                  const unsigned long long *__restrict__ n, uint64_t cap, DevTable t, int max_probes,
                                  uint64_t *__restrict__ ovf_keys, uint32_t *__restrict__ ovf_cnt, uint64_t ovf_cap,
                                  unsigned long long *__restrict__ counters, unsigned long long *__restrict__ distinct) {
    const uint64_t m = *n;
    if (m > cap) return;
    uint32_t added = 0;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < m; i += (uint64_t)gridDim.x * blockDim.x) {
        if (!tbl_add_new(t, keys[i], cnt[i], max_probes, &added)) {
            const unsigned long long j = atomicAdd(&counters[0], 1ULL);
            if (j < ovf_cap) { ovf_keys[j] = keys[i]; ovf_cnt[j] = cnt[i]; }
        }
    }
    added = warp_sum(added);
    if (lane_id() == 0 && added) atomicAdd(distinct, (unsigned long long)added);
}

__global__ void k_fill_empty(Slot *slots, uint64_t cap, uint64_t init_val) {
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < cap; i += (uint64_t)gridDim.x * blockDim.x) {
        ulonglong2 v;
        v.x = EMPTY_KEY;
        v.y = init_val;
        reinterpret_cast<ulonglong2 *>(slots)[i] = v;
    }
}

__global__ void k_occupied(const Slot *__restrict__ slots, uint64_t cap, unsigned long long *out) {
    uint32_t n = 0;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < cap; i += (uint64_t)gridDim.x * blockDim.x)
        n += __ldcs(&slots[i].key) != EMPTY_KEY;
    n = warp_sum(n);
    if (lane_id() == 0 && n) atomicAdd(out, (unsigned long long)n);
}

// K3: keys with count >= min_count.  A block takes a chunk of CP_ITEMS slots
// per thread, ranks its selected slots with a block scan and reserves their
// output range with one atomicAdd per chunk (a per-warp counter atomic on one
// address serialises in L2 on a 2G-slot table).  Output order is fixed by the
// sort that follows.  Bound by memory: 8.6 GB 1.35 ms (256 threads with 16 slots
// each, 32 of an SM's warps, 1.53).
constexpr int CP_THREADS = 512;
constexpr int CP_ITEMS = 4;

__global__ void __launch_bounds__(CP_THREADS) k_compact(const Slot *__restrict__ slots, uint64_t cap, uint32_t min_count,
                                                 uint64_t *__restrict__ okeys, uint32_t *__restrict__ ovals,
                                                 unsigned long long *__restrict__ n_out) {
    __shared__ uint32_t sm[CP_THREADS / 32 + 1];
    __shared__ unsigned long long s_base;
    constexpr uint64_t chunk = (uint64_t)CP_THREADS * CP_ITEMS;
    for (uint64_t base = (uint64_t)blockIdx.x * chunk; base < cap; base += (uint64_t)gridDim.x * chunk) {
        ulonglong2 v[CP_ITEMS];
        uint32_t nsel = 0;
#pragma unroll
        for (int j = 0; j < CP_ITEMS; j++) {
            const uint64_t i = base + (uint64_t)j * CP_THREADS + threadIdx.x;   // coalesced, striped
            v[j].x = EMPTY_KEY;
            v[j].y = 0;
            if (i < cap) v[j] = __ldcs(reinterpret_cast<const ulonglong2 *>(&slots[i]));
            nsel += v[j].x != EMPTY_KEY && (uint32_t)v[j].y >= min_count;
        }
        uint32_t tot;
        uint32_t pre = block_excl_scan<uint32_t>(nsel, sm, &tot);
        if (tot == 0) continue;                   // uniform over the block
        if (threadIdx.x == 0) s_base = atomicAdd(n_out, (unsigned long long)tot);
        __syncthreads();
        uint64_t o = s_base + pre;
#pragma unroll
        for (int j = 0; j < CP_ITEMS; j++) {
            if (v[j].x != EMPTY_KEY && (uint32_t)v[j].y >= min_count) {
                okeys[o] = v[j].x;
                ovals[o] = (uint32_t)v[j].y;
                o++;
            }
        }
        __syncthreads();
    }
}

// jellyfish histo bins: [0] below low, [1 + c - low], [nb - 1] above high.  A
// thread takes HS_ITEMS slots at a time (their loads together) and counts the
// k-mers seen once, most of a table's, in a register.  Bound by memory: one
// read of the table.  8.6 GB: 1.18 ms (a slot at a time, 512 threads, 1.90; 512
// threads with 8 slots 1.87, 512 with 4 in four blocks 1.54).
constexpr int HS_THREADS = 1024;
constexpr int HS_ITEMS = 4;
__global__ void __launch_bounds__(HS_THREADS) k_histo(const Slot *__restrict__ slots, uint64_t cap, uint64_t low, uint64_t high,
                                                      unsigned long long *__restrict__ hist, int use_smem) {
    extern __shared__ uint32_t sh[];
    const uint64_t nb = high - low + 3;
    auto bin_of_count = [&](uint64_t c) { return c < low ? 0 : (c > high ? nb - 1 : 1 + c - low); };
    if (use_smem) {
        for (uint64_t i = threadIdx.x; i < nb; i += HS_THREADS) sh[i] = 0;
        __syncthreads();
    }
    uint32_t once = 0;
    const uint64_t chunk = (uint64_t)HS_THREADS * HS_ITEMS;
    for (uint64_t base = (uint64_t)blockIdx.x * chunk; base < cap; base += (uint64_t)gridDim.x * chunk) {
        ulonglong2 v[HS_ITEMS];
#pragma unroll
        for (int j = 0; j < HS_ITEMS; j++) {
            const uint64_t i = base + (uint64_t)j * HS_THREADS + threadIdx.x;
            v[j].x = EMPTY_KEY;
            if (i < cap) v[j] = __ldcs(reinterpret_cast<const ulonglong2 *>(&slots[i]));
        }
#pragma unroll
        for (int j = 0; j < HS_ITEMS; j++) {
            if (v[j].x == EMPTY_KEY) continue;
            const uint32_t c = (uint32_t)v[j].y;
            if (c == 1) once++;
            else if (use_smem) atomicAdd(&sh[bin_of_count(c)], 1u);
            else atomicAdd(&hist[bin_of_count(c)], 1ULL);
        }
    }
    once = warp_sum(once);
    if (lane_id() == 0 && once) {
        if (use_smem) atomicAdd(&sh[bin_of_count(1)], once);
        else atomicAdd(&hist[bin_of_count(1)], (unsigned long long)once);
    }
    if (use_smem) {
        __syncthreads();
        for (uint64_t i = threadIdx.x; i < nb; i += HS_THREADS)
            if (sh[i]) atomicAdd(&hist[i], (unsigned long long)sh[i]);
    }
}

// K4: each thread formats one record into the block's shared-memory buffer,
// then the block stores its records' bytes in aligned 16-byte pieces.  Bound by
// the formatting's instructions (issue slots 70% busy) and memory (53%).  The
// block scans its records' lengths itself, so that only its first record's place
// comes from memory: 22M records 0.265 ms and 0.066 for the scan of the lengths;
// with a place for every record 0.243 and 0.137.  (With a lane's letters stored
// one by one and a warp's text leaving byte by byte 0.38.)
constexpr int DW_THREADS = DUMP_BLOCK;
constexpr int DW_BYTES = (DW_THREADS * (3 + 10 + MAX_K) + 16 + 15) & ~15;

__global__ void __launch_bounds__(DW_THREADS) k_dump_write(const uint64_t *__restrict__ keys,
                                                          const uint32_t *__restrict__ cnt,
                                                          const uint64_t *__restrict__ off, uint64_t n, int k,
                                                          char *__restrict__ out) {
    __shared__ __align__(16) char buf[DW_BYTES];
    __shared__ uint32_t sm[DW_THREADS / 32 + 1];
    const uint64_t i = (uint64_t)blockIdx.x * DW_THREADS + threadIdx.x;
    const uint64_t w0 = off[blockIdx.x];
    const uint32_t c = i < n ? cnt[i] : 0u, d = dec_digits(c);
    uint32_t bytes;
    const uint32_t at = block_excl_scan<uint32_t>(i < n ? 3u + d + (uint32_t)k : 0u, sm, &bytes);
    if (i < n) {
        char *p = buf + (w0 & 15) + at;
        *p++ = '>';
        p = put_dec(p, c, d);
        *p++ = '\n';
        put_kmer_line(p, keys[i], k);
    }
    __syncthreads();
    block_store(buf, out, w0, bytes);
}

// dump records parsed as reads: name = decimal count, sequence = k-mer, cut
// from the read set's 2-bit codes (the catalogue of 400,000 reads 46 us, byte by byte from the
// letters 112)
__global__ void k_load_dump(const char *__restrict__ text, const uint64_t *__restrict__ name_off,
                            const uint32_t *__restrict__ name_len, const uint64_t *__restrict__ codes,
                            const uint32_t *__restrict__ inv, const uint64_t *__restrict__ rd_off, uint64_t n, int k,
                            int canonical,
                            uint64_t *__restrict__ keys, uint32_t *__restrict__ cnt, uint32_t *__restrict__ err) {
    uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const char *h = text + name_off[i];
    uint32_t hl = name_len[i];
    uint64_t c = 0;
    bool bad = hl == 0;
    for (uint32_t j = 0; j < hl; j++) {
        uint32_t d = (uint8_t)h[j] - (uint32_t)'0';
        if (d > 9) { bad = true; break; }
        c = c * 10 + d;
        if (c > 0xFFFFFFFFull) c = 0xFFFFFFFFull;
    }
    uint64_t s = rd_off[i], L = rd_off[i + 1] - s - 1;
    if (L != (uint64_t)k) bad = true;
    uint64_t fw = 0;
    if (!bad) {
        // the 32 positions from s on; the set's words go on past its last position
        const uint64_t w = s >> 5;
        const uint32_t o = (uint32_t)s & 31u;
        const uint64_t x = o ? (__ldg(codes + w) << (2 * o)) | (__ldg(codes + w + 1) >> (64 - 2 * o)) : __ldg(codes + w);
        bad = __funnelshift_l(__ldg(inv + w + 1), __ldg(inv + w), o) >> (32 - k) != 0u;
        fw = x >> (64 - 2 * k);
    }
    if (bad) {
        atomicExch(&err[DE_PARSE], 1u);
        atomicMin(&err[DE_PARSE + 1], (uint32_t)min((uint64_t)0xFFFFFFFEull, i + 1));
        keys[i] = EMPTY_KEY;
        cnt[i] = 0;
        return;
    }
    keys[i] = canonical ? min(fw, kmer_revcomp(fw, k)) : fw;
    cnt[i] = (uint32_t)c;
}

static inline unsigned grid_for(uint64_t n, int threads) { return (unsigned)((n + threads - 1) / threads); }

static unsigned stream_grid(tk_ctx *c, uint64_t n, int threads) {
    uint64_t g = (n + threads - 1) / threads;
    uint64_t cap = (uint64_t)c->sm_count * 8;
    return (unsigned)std::max<uint64_t>(1, std::min(g, cap));
}

// ------------------------------------------------------------------ host side

// fill = false leaves the slots unwritten: the partitioned count pass fills
// each slice right before its inserts (a "fresh" table)
static int table_alloc_geom(tk_table *t, uint64_t capacity, uint64_t init_val, bool fill) {
    tk_ctx *c = t->ctx;
    Slot *s = nullptr;
    TK_TRY(dmalloc(c, (void **)&s, capacity * sizeof(Slot), "k-mer table"));
    if (fill) {
        k_fill_empty<<<stream_grid(c, capacity, 256), 256, 0, c->stream>>>(s, capacity, init_val);
        c->launches++;
    }
    t->fresh = !fill;
    int bits = 0;
    while ((1ULL << bits) < capacity) bits++;
    int lbits = std::min(bits, MAX_LBITS);
    if (bits - lbits > BUCKET_BITS) lbits = bits - BUCKET_BITS;   // > 2^33 slots: larger partitions
    t->t.slots = s;
    t->t.lbits = lbits;
    t->t.pbits = bits - lbits;
    t->t.lmask = (1ULL << lbits) - 1;
    t->capacity = capacity;
    return check_launch(c, "table fill");
}

// n empty slots whose value words are init_val
void table_fill_empty(tk_ctx *c, Slot *slots, uint64_t n, uint64_t init_val) {
    k_fill_empty<<<stream_grid(c, n, 256), 256, 0, c->stream>>>(slots, n, init_val);
    c->launches++;
}

int table_alloc_init(tk_table *t, uint64_t capacity, uint64_t init_val) {
    return table_alloc_geom(t, capacity, init_val, true);
}

int table_alloc(tk_table *t, uint64_t capacity) { return table_alloc_geom(t, capacity, 0, true); }

static int overflow_reset(tk_table *t) {
    return cuda_check(t->ctx, cudaMemsetAsync(t->d_counters, 0, sizeof(unsigned long long), t->ctx->stream), "ovf reset");
}

static int overflow_read(tk_table *t, unsigned long long *n) {
    tk_ctx *c = t->ctx;
    TK_CUDA(c, cudaMemcpyAsync(n, t->d_counters, sizeof(unsigned long long), cudaMemcpyDeviceToHost, c->stream));
    TK_CUDA(c, cudaStreamSynchronize(c->stream));
    return TK_OK;
}

// Moves every entry to a table of new_capacity slots.
int table_rehash(tk_table *t, uint64_t new_capacity) {
    tk_ctx *c = t->ctx;
    for (int attempt = 0; attempt < 8; attempt++) {
        Slot *old = t->t.slots;
        const DevTable old_t = t->t;
        uint64_t old_cap = t->capacity;
        TK_TRY(table_alloc(t, new_capacity));
        TK_TRY(overflow_reset(t));
        if (old) {
            k_rehash<<<stream_grid(c, old_cap, 256), 256, 0, c->stream>>>(old, old_cap, t->t, c->max_probes, t->d_ovf,
                                                                           (uint32_t *)(t->d_ovf + t->ovf_cap), t->ovf_cap,
                                                                           t->d_counters);
            c->launches++;
        }
        unsigned long long ovf = 0;
        TK_TRY(overflow_read(t, &ovf));
        if (ovf == 0) {
            dfree(c, old);
            return TK_OK;
        }
        // a probe run too long even in the larger table: go bigger from the old copy
        dfree(c, t->t.slots);
        t->t = old_t;
        t->capacity = old_cap;
        new_capacity *= 2;
    }
    return set_err(c, TK_E_TABLE_FULL, "rehash could not place every key");
}

// Re-inserts the overflow list after doubling the table, until it drains.
static int drain_overflow(tk_table *t) {
    tk_ctx *c = t->ctx;
    for (int round = 0; round < 8; round++) {
        unsigned long long ovf = 0;
        TK_TRY(overflow_read(t, &ovf));
        if (ovf == 0) return TK_OK;
        t->distinct_valid = false;
        if (ovf > t->ovf_cap)
            return set_err(c, TK_E_TABLE_FULL,
                           "table overflow list overran (" + std::to_string(ovf) + " keys); create the table with a larger capacity");
        // copy the pending pairs aside, grow, and insert them
        uint64_t *pk = nullptr;
        uint32_t *pc = nullptr;
        TK_TRY(dmalloc(c, (void **)&pk, ovf * 8, "overflow keys"));
        int e = dmalloc(c, (void **)&pc, ovf * 4, "overflow counts");
        if (!e) {
            cudaMemcpyAsync(pk, t->d_ovf, ovf * 8, cudaMemcpyDeviceToDevice, c->stream);
            cudaMemcpyAsync(pc, t->d_ovf + t->ovf_cap, ovf * 4, cudaMemcpyDeviceToDevice, c->stream);
            e = table_rehash(t, t->capacity * 2);
        }
        if (!e) e = overflow_reset(t);
        if (!e) {
            k_insert_pairs<<<stream_grid(c, ovf, 256), 256, 0, c->stream>>>(pk, pc, ovf, t->t, c->max_probes, t->d_ovf,
                                                                             (uint32_t *)(t->d_ovf + t->ovf_cap), t->ovf_cap,
                                                                             t->d_counters);
            c->launches++;
            e = check_launch(c, "overflow insert");
        }
        dfree(c, pk);
        dfree(c, pc);
        if (e) return e;
    }
    return set_err(c, TK_E_TABLE_FULL, "overflow did not drain");
}

static double hll_estimate(const uint32_t *regs) {
    double sum = 0;
    int zeros = 0;
    for (int i = 0; i < HLL_M; i++) {
        sum += std::ldexp(1.0, -(int)regs[i]);
        zeros += regs[i] == 0;
    }
    double m = HLL_M, alpha = 0.7213 / (1.0 + 1.079 / m);
    double est = alpha * m * m / sum;
    if (est <= 2.5 * m && zeros) est = m * std::log(m / zeros);
    return est;
}

static uint64_t pow2_at_least(uint64_t x) {
    uint64_t p = 1024;
    while (p < x) p <<= 1;
    return p;
}

// Pass 2 with global atomics, one partition after another: a launch prepares
// slice p (fills a fresh slice, or prefetches a filled one to L2), then a
// launch CAS-probes and adds partition p's keys into it.  Preparing slice p+1
// inside the insert of p instead (the writes of one slice competing in L2 with
// the atomics on the other) measured ~12% slower.
static int count_by_atomics(tk_table *t, const std::vector<BucketKeys> &bk) {
    tk_ctx *c = t->ctx;
    const int nparts = 1 << t->t.pbits;
    const int mode = t->fresh ? NEXT_FILL : (t->t.pbits > 0 ? NEXT_PREFETCH : NEXT_NONE);
    const unsigned igrid = (unsigned)c->sm_count * 8;
    for (int p = 0; p < nparts; p++) {
        if (mode != NEXT_NONE) {   // slice p filled (fresh) or prefetched once, then every set's keys of partition p
            k_part_step<<<igrid, CT_THREADS, 0, c->stream>>>(bk[0].keys, bk[0].offs, bk[0].cols, -1, p, t->t, mode,
                                                             c->max_probes, t->d_ovf, (uint32_t *)(t->d_ovf + t->ovf_cap),
                                                             t->ovf_cap, t->d_counters);
            c->launches++;
        }
        for (const BucketKeys &b : bk) {
            if (!b.keys) continue;
            k_part_step<<<igrid, CT_THREADS, 0, c->stream>>>(b.keys, b.offs, b.cols, p, -1, t->t, mode, c->max_probes,
                                                             t->d_ovf, (uint32_t *)(t->d_ovf + t->ovf_cap), t->ovf_cap,
                                                             t->d_counters);
            c->launches++;
        }
    }
    return check_launch(c, "count insert");
}

// Pass 2 by ranges on a fresh table (see k_sr_build).  *done is false when
// the deferred list overran its capacity: the table is then emptied again and
// the caller counts with count_by_atomics instead, so nothing is lost.
static int count_by_ranges(tk_table *t, const std::vector<BucketKeys> &bk, const std::vector<const uint64_t *> &starts_of,
                           bool *done, bool *overflowed) {
    tk_ctx *c = t->ctx;
    *done = false;
    const int nparts = 1 << t->t.pbits;
    // ranges per slice: SR_BUILD_PER_SM per SM, more if a range would not fit in shared memory
    const uint64_t slice = 1ULL << t->t.lbits, wave = (uint64_t)c->sm_count * SR_BUILD_PER_SM;
    uint32_t nsub;
    if (slice / 1024 < wave) nsub = (uint32_t)(slice / 1024);   // a small slice: ranges of 1024 slots
    else nsub = (uint32_t)(wave * ((slice + wave * SR_MAX_SLOTS - 1) / (wave * SR_MAX_SLOTS)));
    if (nsub > 0xFFFF) return TK_OK;   // run starts and ranges are 16-bit
    const uint64_t bpp = (uint64_t)(NBUCKETS >> t->t.pbits);
    const uint32_t nsets = (uint32_t)bk.size();
    std::vector<KeySeg> segs((size_t)nparts * nsets);
    std::vector<PartGeom> parts(nparts);
    std::vector<int> batch{0};                 // first partition of every batch, then nparts
    uint64_t all_keys = 0, batch_keys = 0, batch_chunks = 0, max_chunks = 0;
    for (int p = 0; p < nparts; p++) {
        uint64_t part = 0;
        for (uint32_t q = 0; q < nsets; q++) {
            KeySeg &g = segs[(size_t)p * nsets + q];
            // partition p's keys are one segment of each set's buffer
            const uint64_t *b = starts_of[q];
            g.keys = bk[q].keys ? bk[q].keys + b[p * bpp] : nullptr;
            g.len = bk[q].keys ? b[(p + 1) * bpp] - b[p * bpp] : 0;
            part += g.len;
        }
        if (p > batch.back() && batch_keys + part > SR_BATCH_KEYS) {
            batch.push_back(p);
            batch_keys = batch_chunks = 0;
        }
        const uint64_t chunks = (part + SG_CHUNK - 1) / SG_CHUNK;
        parts[p].chunk0 = (uint32_t)batch_chunks;
        parts[p].chunks = (uint32_t)chunks;
        batch_keys += part;
        batch_chunks += chunks;
        max_chunks = std::max(max_chunks, batch_chunks);
        all_keys += part;
    }
    batch.push_back(nparts);
    uint64_t defer_cap = std::max<uint64_t>(1u << 16, std::min<uint64_t>(all_keys / 64, 1u << 24));
    if (const char *v = getenv("TRINKMER_DEFER_CAP")) defer_cap = std::max<uint64_t>(1, strtoull(v, nullptr, 10));   // tests: force the fallback
    uint64_t *grouped = nullptr, *defer_keys = nullptr;
    uint32_t *defer_cnt = nullptr;
    uint16_t *starts = nullptr;
    unsigned long long *counters = nullptr;   // deferred keys, distinct keys
    KeySeg *d_segs = nullptr;
    PartGeom *d_parts = nullptr;
    int e = dmalloc(c, (void **)&grouped, max_chunks * SG_CHUNK * 8, "grouped keys");
    if (!e) e = dmalloc(c, (void **)&starts, max_chunks * (nsub + 1) * 2, "group starts");
    if (!e) e = dmalloc(c, (void **)&d_segs, segs.size() * sizeof(KeySeg), "partition segments");
    if (!e) e = dmalloc(c, (void **)&d_parts, parts.size() * sizeof(PartGeom), "partition chunks");
    if (!e) e = dmalloc(c, (void **)&defer_keys, defer_cap * 8, "deferred keys");
    if (!e) e = dmalloc(c, (void **)&defer_cnt, defer_cap * 4, "deferred counts");
    if (!e) e = dmalloc(c, (void **)&counters, 16, "count counters");
    if (e == TK_E_OOM) {   // no room for the batches: the caller counts with atomics, which need none
        if (grouped) dfree(c, grouped);
        if (starts) dfree(c, starts);
        if (d_segs) dfree(c, d_segs);
        if (d_parts) dfree(c, d_parts);
        if (defer_keys) dfree(c, defer_keys);
        if (defer_cnt) dfree(c, defer_cnt);
        return TK_OK;
    }
    if (!e) e = cuda_check(c, cudaMemcpyAsync(d_segs, segs.data(), segs.size() * sizeof(KeySeg), cudaMemcpyHostToDevice,
                                              c->stream), "partition segments h2d");
    if (!e) e = cuda_check(c, cudaMemcpyAsync(d_parts, parts.data(), parts.size() * sizeof(PartGeom), cudaMemcpyHostToDevice,
                                              c->stream), "partition chunks h2d");
    if (!e) e = cuda_check(c, cudaMemsetAsync(counters, 0, 16, c->stream), "count counters reset");
    const int group_smem = (int)(SG_CHUNK * 8 + nsub * 4), build_smem = (int)sizeof(BuildSmem);
    if (!e) e = cuda_check(c, cudaFuncSetAttribute(k_sr_build, cudaFuncAttributeMaxDynamicSharedMemorySize, build_smem),
                           "range build smem");
    if (!e) e = cuda_check(c, cudaFuncSetAttribute(k_sr_group, cudaFuncAttributeMaxDynamicSharedMemorySize, group_smem),
                           "range group smem");
    for (size_t b = 0; !e && b + 1 < batch.size(); b++) {
        const int p0 = batch[b], np = batch[b + 1] - p0;
        const unsigned chunks = parts[p0 + np - 1].chunk0 + parts[p0 + np - 1].chunks;
        if (chunks) {
            k_sr_group<<<chunks, SG_THREADS, group_smem, c->stream>>>(d_segs + (size_t)p0 * nsets, nsets, d_parts + p0, np, t->t,
                                                                     nsub, grouped, starts);
            c->launches++;
        }
        k_sr_build<<<nsub * np, SR_BUILD_THREADS, build_smem, c->stream>>>(grouped, starts, d_parts + p0, nsub, p0, t->t,
                                                                          defer_keys, defer_cnt, defer_cap, counters,
                                                                          counters + 1);
        c->launches++;
    }
    if (!e) {
        k_insert_deferred<<<(unsigned)c->sm_count * 8, 256, 0, c->stream>>>(defer_keys, defer_cnt, counters, defer_cap, t->t,
                                                                      c->max_probes, t->d_ovf,
                                                                      (uint32_t *)(t->d_ovf + t->ovf_cap), t->ovf_cap,
                                                                      t->d_counters, counters + 1);
        c->launches++;
        e = check_launch(c, "range build");
    }
    // deferred keys, distinct keys, keys on the overflow list
    volatile unsigned long long *h = reinterpret_cast<volatile unsigned long long *>(c->h_stage);
    if (!e) e = cuda_check(c, cudaMemcpyAsync(c->h_stage, counters, 16, cudaMemcpyDeviceToHost, c->stream), "count counters d2h");
    if (!e) e = cuda_check(c, cudaMemcpyAsync(c->h_stage + 16, t->d_counters, 8, cudaMemcpyDeviceToHost, c->stream), "overflow d2h");
    if (!e) e = cuda_check(c, cudaStreamSynchronize(c->stream), "count sync");
    if (!e && h[0] > defer_cap) {
        // the deferred list overran: empty the table again and count with atomics
        k_fill_empty<<<stream_grid(c, t->capacity, 256), 256, 0, c->stream>>>(t->t.slots, t->capacity, 0);
        c->launches++;
        t->fresh = false;
        e = check_launch(c, "table refill");
    } else if (!e) {
        t->fresh = false;
        t->distinct = h[1];   // every key of the table was new to it once
        t->distinct_valid = true;
        *overflowed = h[2] != 0;
        *done = true;
    }
    if (grouped) dfree(c, grouped);
    if (starts) dfree(c, starts);
    if (d_segs) dfree(c, d_segs);
    if (d_parts) dfree(c, d_parts);
    if (defer_keys) dfree(c, defer_keys);
    if (defer_cnt) dfree(c, defer_cnt);
    if (counters) dfree(c, counters);
    return e;
}

// where each of the NBUCKETS buckets begins, and where the last one ends
__global__ void k_bucket_starts(const uint64_t *__restrict__ offs, uint64_t cols, uint64_t *__restrict__ starts) {
    const uint32_t b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b <= NBUCKETS) starts[b] = offs[(uint64_t)b * cols];
}

// Pass 1 for one read set: the bucket histogram of its windows with the HLL
// sketch (a union into t->d_hll) and the window count (added to
// t->d_counters[1]), then its windows into a key buffer of its own, bucket
// by bucket.  The two kernels use one fixed grid, so every tile goes to the
// same block (histogram column) in both.
int table_bucket_pass(tk_table *t, const tk_reads *r, BucketKeys *out) {
    tk_ctx *c = t->ctx;
    *out = BucketKeys();
    const uint64_t len = r->seq_len;
    if (len == 0) return TK_OK;
    const uint64_t tile = SC_TILE;
    const unsigned grid = (unsigned)std::max<uint64_t>(1, std::min<uint64_t>((len + tile - 1) / tile, (uint64_t)c->sm_count));
    const uint64_t cols = grid, cells = (uint64_t)NBUCKETS * cols;
    uint32_t *hist = nullptr;
    uint64_t *offs = nullptr, *keys = nullptr;
    TK_TRY(dmalloc(c, (void **)&hist, cells * 4, "bucket histogram"));
    int e = dmalloc(c, (void **)&offs, (cells + 1) * 8, "bucket offsets");
    cudaEvent_t ev;
    if (!e) {
        prof_begin(c, TK_KID_HLL, &ev);
        if (t->canonical)
            k_part_hist<true><<<grid, HIST_THREADS, 0, c->stream>>>(r->d_codes, r->d_inv, len, t->k, hist, cols, 0,
                                                                  t->d_hll, t->d_counters + 1);
        else
            k_part_hist<false><<<grid, HIST_THREADS, 0, c->stream>>>(r->d_codes, r->d_inv, len, t->k, hist, cols, 0,
                                                                   t->d_hll, t->d_counters + 1);
        c->launches++;
        prof_end(c, TK_KID_HLL, ev, len);
        e = check_launch(c, "bucket histogram");
    }
    // key-buffer entries: the windows plus the EMPTY_KEY padding of every
    // region (0 exactly when the set has no windows).  A set of up to SC_SMALL
    // positions gets room for a window at each of them instead and is not
    // waited for, unless that much memory is not to be had.
    uint64_t padded = len + 3 * cells;
    uint64_t *starts = nullptr;
    if (!e) e = dmalloc(c, (void **)&starts, (NBUCKETS + 1) * 8, "bucket starts");
    if (!e && len <= SC_SMALL && dmalloc(c, (void **)&keys, padded * 8, "bucketed k-mers") == TK_OK) {
        e = scan_excl_u32_to_u64_async(c, hist, offs, cells, offs + cells);
    } else if (!e) {
        e = scan_excl_u32_to_u64(c, hist, offs, cells, &padded);   // synchronises
        if (!e) e = cuda_check(c, cudaMemcpyAsync(offs + cells, &padded, 8, cudaMemcpyHostToDevice, c->stream), "bucket end");
        if (!e && padded) e = dmalloc(c, (void **)&keys, padded * 8, "bucketed k-mers");
    }
    if (!e && padded) {
        k_bucket_starts<<<(NBUCKETS + 256) / 256, 256, 0, c->stream>>>(offs, cols, starts);
        c->launches++;
        static_assert(SC_SMEM <= 227 * 1024, "bucket staging exceeds shared memory");
        if (!e) e = cuda_check(c, cudaFuncSetAttribute(k_part_scatter<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                       (int)SC_SMEM), "scatter smem");
        if (!e) e = cuda_check(c, cudaFuncSetAttribute(k_part_scatter<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                       (int)SC_SMEM), "scatter smem");
        if (!e) {
            prof_begin(c, TK_KID_SCATTER, &ev);
            if (t->canonical)
                k_part_scatter<true><<<grid, SC_THREADS, SC_SMEM, c->stream>>>(r->d_codes, r->d_inv, len, t->k, offs, cols,
                                                                              0, keys, c->d_err + DE_COUNT);
            else
                k_part_scatter<false><<<grid, SC_THREADS, SC_SMEM, c->stream>>>(r->d_codes, r->d_inv, len, t->k, offs, cols,
                                                                               0, keys, c->d_err + DE_COUNT);
            c->launches++;
            prof_end(c, TK_KID_SCATTER, ev, padded);
            e = check_launch(c, "bucket scatter");
        }
    }
    dfree(c, hist);
    if (e || !padded) {
        if (keys) dfree(c, keys);
        if (offs) dfree(c, offs);
        if (starts) dfree(c, starts);
        return e;
    }
    out->keys = keys;
    out->offs = offs;
    out->starts = starts;
    out->cols = cols;
    return TK_OK;
}

void table_bucket_free(tk_table *t, BucketKeys *bk) {
    if (bk->keys) dfree(t->ctx, bk->keys);
    if (bk->offs) dfree(t->ctx, bk->offs);
    if (bk->starts) dfree(t->ctx, bk->starts);
    *bk = BucketKeys();
}

// Pass 2 for the sets whose pass 1 ran since the window counter was reset:
// the table sized from the HLL sketch (allocated fresh, or grown), then every
// set's keys counted partition by partition; frees the key buffers.
int table_count_buckets(tk_table *t, std::vector<BucketKeys> &bk) {
    tk_ctx *c = t->ctx;
    // the sketch, the window count and every set's bucket starts, read back at
    // one synchronisation through the context's page-locked stage (the starts of
    // more sets than fit there through pageable memory)
    constexpr size_t STARTS = (NBUCKETS + 1) * 8, STAGED = (STAGE_BYTES - HLL_M * 4 - 8) / STARTS;
    uint64_t windows = 0;
    std::vector<uint32_t> regs(HLL_M);
    std::vector<uint64_t> starts(bk.size() * (NBUCKETS + 1));
    std::vector<const uint64_t *> starts_of(bk.size());
    int e = cuda_check(c, cudaMemcpyAsync(c->h_stage, t->d_hll, HLL_M * 4, cudaMemcpyDeviceToHost, c->stream), "hll d2h");
    if (!e) e = cuda_check(c, cudaMemcpyAsync(c->h_stage + HLL_M * 4, t->d_counters + 1, 8, cudaMemcpyDeviceToHost, c->stream),
                           "window count d2h");
    for (size_t q = 0; q < bk.size() && !e; q++) {
        void *to = q < STAGED ? (void *)(c->h_stage + HLL_M * 4 + 8 + q * STARTS) : (void *)(starts.data() + q * (NBUCKETS + 1));
        if (bk[q].keys) e = cuda_check(c, cudaMemcpyAsync(to, bk[q].starts, STARTS, cudaMemcpyDeviceToHost, c->stream), "bucket starts d2h");
    }
    if (!e) e = cuda_check(c, cudaStreamSynchronize(c->stream), "hll sync");
    if (!e) e = wait_status(c);
    if (!e) {
        memcpy(regs.data(), c->h_stage, HLL_M * 4);
        memcpy(&windows, c->h_stage + HLL_M * 4, 8);
        for (size_t q = 0; q < bk.size(); q++) {
            uint64_t *at = starts.data() + q * (NBUCKETS + 1);
            if (q < STAGED && bk[q].keys) memcpy(at, c->h_stage + HLL_M * 4 + 8 + q * STARTS, STARTS);
            starts_of[q] = at;
        }
    }
    if (!e) {
        double est = hll_estimate(regs.data());
        uint64_t want = pow2_at_least((uint64_t)(est * 1.08 / t->max_load) + 1);
        if (t->capacity == 0) e = table_alloc_geom(t, want, 0, false);   // fresh: filled slice by slice below
        else if (want > t->capacity) e = table_rehash(t, want);
    }
    cudaEvent_t ev;
    bool settled = false;   // nothing on the overflow list, as read back already
    if (!e && windows) {
        e = overflow_reset(t);
        t->distinct_valid = false;
        prof_begin(c, TK_KID_COUNT, &ev);
        bool done = false, overflowed = true;
        if (!e && t->fresh && t->t.lbits >= SR_MIN_LBITS) e = count_by_ranges(t, bk, starts_of, &done, &overflowed);
        if (!e && !done) e = count_by_atomics(t, bk);
        prof_end(c, TK_KID_COUNT, ev, windows);
        if (!e) e = check_launch(c, "count insert");
        if (!e) t->fresh = false;
        settled = done && !overflowed;
    } else if (!e && t->fresh) {
        // nothing to insert: still leave every slot empty
        k_fill_empty<<<stream_grid(c, t->capacity, 256), 256, 0, c->stream>>>(t->t.slots, t->capacity, 0);
        c->launches++;
        t->fresh = false;
        e = check_launch(c, "table fill");
    }
    for (BucketKeys &b : bk) table_bucket_free(t, &b);
    if (e && t->fresh && t->t.slots) {
        // a failed first pass must not leave unwritten slots behind
        k_fill_empty<<<stream_grid(c, t->capacity, 256), 256, 0, c->stream>>>(t->t.slots, t->capacity, 0);
        c->launches++;
        t->fresh = false;
    }
    if (e) return e;
    t->total += windows;
    return settled ? TK_OK : drain_overflow(t);
}

// Resets the window counter before a group of pass-1 calls.
int table_count_begin(tk_table *t) {
    return cuda_check(t->ctx, cudaMemsetAsync(t->d_counters + 1, 0, 8, t->ctx->stream), "window counter");
}

// Counts every window of one or more packed read arrays into the table: pass
// 1 per set, then one partitioned pass 2 over all of them (the table is
// touched once for all of them); sets beyond MAX_KEY_SEGS are counted in
// further groups.
int table_count_many(tk_table *t, const tk_reads *const *sets, int nsets) {
    for (int g0 = 0; g0 < nsets; g0 += MAX_KEY_SEGS) {
        const int g1 = std::min(nsets, g0 + MAX_KEY_SEGS);
        uint64_t total_len = 0;
        for (int s = g0; s < g1; s++) total_len += sets[s]->seq_len;
        if (total_len == 0) continue;
        TK_TRY(table_count_begin(t));
        std::vector<BucketKeys> bk(g1 - g0);
        int e = TK_OK;
        for (int s = g0; s < g1 && !e; s++) e = table_bucket_pass(t, sets[s], &bk[s - g0]);
        if (e) {
            for (BucketKeys &b : bk) table_bucket_free(t, &b);
            return e;
        }
        TK_TRY(table_count_buckets(t, bk));
    }
    return TK_OK;
}

int table_count_seq(tk_table *t, const tk_reads *r) { return table_count_many(t, &r, 1); }

static int table_distinct(tk_table *t) {
    tk_ctx *c = t->ctx;
    if (t->distinct_valid) return TK_OK;
    if (!t->capacity) {
        t->distinct = 0;
        t->distinct_valid = true;
        return TK_OK;
    }
    unsigned long long *d = nullptr, h = 0;
    TK_TRY(dmalloc(c, (void **)&d, 8, "occupied"));
    cudaMemsetAsync(d, 0, 8, c->stream);
    k_occupied<<<stream_grid(c, t->capacity, 256), 256, 0, c->stream>>>(t->t.slots, t->capacity, d);
    c->launches++;
    int e = cuda_check(c, cudaMemcpyAsync(&h, d, 8, cudaMemcpyDeviceToHost, c->stream), "occupied d2h");
    if (!e) e = cuda_check(c, cudaStreamSynchronize(c->stream), "occupied sync");
    dfree(c, d);
    if (!e) {
        t->distinct = h;
        t->distinct_valid = true;
    }
    return e;
}

int table_info(tk_table *t, uint64_t *distinct, uint64_t *total, uint64_t *capacity) {
    if (distinct) {
        TK_TRY(table_distinct(t));   // a scan of the table, only when asked for
        *distinct = t->distinct;
    }
    if (total) *total = t->total;
    if (capacity) *capacity = t->capacity;
    return TK_OK;
}

int table_histo(tk_table *t, uint64_t low, uint64_t high, uint64_t *hist) {
    tk_ctx *c = t->ctx;
    if (high < low) return set_err(c, TK_E_INVAL, "histo: high < low");
    uint64_t nb = high - low + 3;
    unsigned long long *d = nullptr;
    TK_TRY(dmalloc(c, (void **)&d, nb * 8, "histo"));
    cudaMemsetAsync(d, 0, nb * 8, c->stream);
    int e = TK_OK;
    if (t->capacity) {
        cudaEvent_t ev;
        prof_begin(c, TK_KID_COMPACT, &ev);
        size_t smem = nb * 4;
        int use_smem = smem <= 96 * 1024;
        if (use_smem && smem > 48 * 1024)
            cudaFuncSetAttribute(k_histo, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        k_histo<<<(unsigned)c->sm_count * 2, HS_THREADS, use_smem ? smem : 0, c->stream>>>(t->t.slots, t->capacity, low, high, d,
                                                                                    use_smem);
        c->launches++;
        prof_end(c, TK_KID_COMPACT, ev, t->capacity);
        e = check_launch(c, "histo");
    }
    if (!e) e = cuda_check(c, cudaMemcpyAsync(hist, d, nb * 8, cudaMemcpyDeviceToHost, c->stream), "histo d2h");
    if (!e) e = cuda_check(c, cudaStreamSynchronize(c->stream), "histo sync");
    dfree(c, d);
    if (!e) {
        // every occupied slot fell in one bin: the bins add up to the distinct k-mers
        uint64_t distinct = 0;
        for (uint64_t i = 0; i < nb; i++) distinct += hist[i];
        t->distinct = distinct;
        t->distinct_valid = true;
    }
    return e;
}

// Sorted (key, count) pairs with count >= min_count into freshly allocated
// device arrays (caller frees with dfree).
int table_sorted_pairs(tk_table *t, uint32_t min_count, uint64_t **keys_out, uint32_t **cnt_out, uint64_t *n_out) {
    tk_ctx *c = t->ctx;
    *keys_out = nullptr;
    *cnt_out = nullptr;
    *n_out = 0;
    TK_TRY(table_distinct(t));
    uint64_t upper = std::max<uint64_t>(t->distinct, 1);
    uint64_t *k0 = nullptr, *k1 = nullptr;
    uint32_t *v0 = nullptr, *v1 = nullptr;
    unsigned long long *d_n = nullptr;
    int e = dmalloc(c, (void **)&k0, upper * 8, "dump keys");
    if (!e) e = dmalloc(c, (void **)&v0, upper * 4, "dump counts");
    if (!e) e = dmalloc(c, (void **)&k1, upper * 8, "dump keys tmp");
    if (!e) e = dmalloc(c, (void **)&v1, upper * 4, "dump counts tmp");
    if (!e) e = dmalloc(c, (void **)&d_n, 8, "dump n");
    unsigned long long hn = 0;
    if (!e && t->capacity) {
        cudaMemsetAsync(d_n, 0, 8, c->stream);
        cudaEvent_t ev;
        prof_begin(c, TK_KID_COMPACT, &ev);
        k_compact<<<(unsigned)std::min<uint64_t>((t->capacity + CP_THREADS * CP_ITEMS - 1) / (CP_THREADS * CP_ITEMS),
                                                   (uint64_t)c->sm_count * 4), CP_THREADS, 0, c->stream>>>(
            t->t.slots, t->capacity, min_count, k0, v0, d_n);
        c->launches++;
        prof_end(c, TK_KID_COMPACT, ev, t->capacity);
        e = cuda_check(c, cudaMemcpyAsync(&hn, d_n, 8, cudaMemcpyDeviceToHost, c->stream), "compact n");
        if (!e) e = cuda_check(c, cudaStreamSynchronize(c->stream), "compact sync");
    }
    bool in_tmp = false;
    if (!e && hn > 1) {
        cudaEvent_t ev;
        prof_begin(c, TK_KID_SORT, &ev);
        e = sort_distinct_pairs(c, k0, v0, hn, 2 * t->k, k1, v1, &in_tmp);
        prof_end(c, TK_KID_SORT, ev, hn);
    }
    if (d_n) dfree(c, d_n);
    if (e) {
        dfree(c, k0); dfree(c, k1); dfree(c, v0); dfree(c, v1);
        return e;
    }
    if (in_tmp) {
        std::swap(k0, k1);
        std::swap(v0, v1);
    }
    dfree(c, k1);
    dfree(c, v1);
    *keys_out = k0;
    *cnt_out = v0;
    *n_out = hn;
    return TK_OK;
}

// K4: format sorted pairs as ">COUNT\nKMER\n" into a device buffer (the low
// 2k bits of each key); with offs_out, the places in the text of every
// DUMP_BLOCK-th record are handed to the caller (its device block to free)
// instead of freed.
int format_dump(tk_ctx *c, const uint64_t *keys, const uint32_t *cnt, uint64_t n, int k, char **text_out,
                uint64_t *len_out, uint64_t **offs_out) {
    *text_out = nullptr;
    *len_out = 0;
    if (offs_out) *offs_out = nullptr;
    if (n == 0) return TK_OK;
    uint64_t *offs = nullptr;
    TK_TRY(dmalloc(c, (void **)&offs, (n + DUMP_BLOCK - 1) / DUMP_BLOCK * 8, "dump offsets"));
    uint64_t total = 0;
    cudaEvent_t ev;
    prof_begin(c, TK_KID_DUMP, &ev);
    int e = scan_record_lengths(c, cnt, offs, n, k, &total);
    char *text = nullptr;
    if (!e) e = dmalloc(c, (void **)&text, total, "dump text");
    if (!e) {
        k_dump_write<<<grid_for(n, DW_THREADS), DW_THREADS, 0, c->stream>>>(keys, cnt, offs, n, k, text);
        c->launches++;
        e = check_launch(c, "dump write");
    }
    prof_end(c, TK_KID_DUMP, ev, n);
    if (e) {
        if (offs) dfree(c, offs);
        if (text) dfree(c, text);
        return e;
    }
    if (offs_out) *offs_out = offs;
    else dfree(c, offs);
    *text_out = text;
    *len_out = total;
    return TK_OK;
}

int table_insert_pairs(tk_table *t, const uint64_t *d_keys, const uint32_t *d_cnt, uint64_t n) {
    tk_ctx *c = t->ctx;
    if (n == 0) return TK_OK;
    TK_TRY(table_distinct(t));
    uint64_t need = pow2_at_least((uint64_t)((double)(t->distinct + n) / t->max_load) + 1);
    if (t->capacity == 0) TK_TRY(table_alloc(t, need));
    else if (need > t->capacity) TK_TRY(table_rehash(t, need));
    TK_TRY(overflow_reset(t));
    cudaEvent_t ev;
    prof_begin(c, TK_KID_LOAD, &ev);
    k_insert_pairs<<<stream_grid(c, n, 256), 256, 0, c->stream>>>(d_keys, d_cnt, n, t->t, c->max_probes, t->d_ovf,
                                                                   (uint32_t *)(t->d_ovf + t->ovf_cap), t->ovf_cap,
                                                                   t->d_counters);
    c->launches++;
    prof_end(c, TK_KID_LOAD, ev, n);
    TK_TRY(check_launch(c, "insert pairs"));
    t->distinct_valid = false;
    return drain_overflow(t);
}

int table_load_dump_reads(tk_table *t, const tk_reads *r) {
    tk_ctx *c = t->ctx;
    uint64_t n = r->n_reads;
    if (n == 0) return TK_OK;
    uint64_t *keys = nullptr;
    uint32_t *cnt = nullptr;
    TK_TRY(dmalloc(c, (void **)&keys, n * 8, "catalogue keys"));
    int e = dmalloc(c, (void **)&cnt, n * 4, "catalogue counts");
    if (!e) e = cuda_check(c, cudaMemsetAsync(c->d_err, 0, DE_COUNT * 4, c->stream), "err reset");
    if (!e) {
        uint32_t big = 0xFFFFFFFFu;
        cudaMemcpyAsync(c->d_err + DE_PARSE + 1, &big, 4, cudaMemcpyHostToDevice, c->stream);
        k_load_dump<<<grid_for(n, 256), 256, 0, c->stream>>>(r->d_text, r->d_name_off, r->d_name_len, r->d_codes, r->d_inv, r->d_rd_off,
                                                             n, t->k, t->canonical, keys, cnt, c->d_err);
        c->launches++;
        uint32_t herr[2] = {0, 0};
        e = cuda_check(c, cudaMemcpyAsync(herr, c->d_err + DE_PARSE, 8, cudaMemcpyDeviceToHost, c->stream), "load err");
        if (!e) e = cuda_check(c, cudaStreamSynchronize(c->stream), "load sync");
        if (!e && herr[0])
            e = set_err(c, TK_E_PARSE, "k-mer catalogue: record " + std::to_string(herr[1]) +
                                           " is not '>COUNT' followed by a " + std::to_string(t->k) + "-mer of A/C/G/T");
    }
    if (!e) e = table_insert_pairs(t, keys, cnt, n);
    dfree(c, keys);
    if (cnt) dfree(c, cnt);
    return e;
}

}  // namespace tk
