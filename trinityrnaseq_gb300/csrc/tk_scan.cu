// tk_scan.cu -- device-wide exclusive scan and LSD radix sort of (u64 key,
// u32 value) pairs.  Both are single-pass streaming kernels: a block takes the
// next tile (a ticket, so that every earlier tile already has a running
// block), publishes what its tile adds, and learns what the earlier tiles add
// up to by walking back over their published words until one of them is a
// complete prefix.  The scan thus reads its input and writes its output once;
// each radix pass reads and writes the pairs once, the digit counts of all
// passes coming from one read of the keys beforehand.
//
// A published word is 64 bits, written and read whole, so it needs no fence:
// bits 62-63 say what it holds (0 nothing yet, 1 the tile alone, 2 the tile
// and all before it) and, in the sort, bits 58-61 the pass it belongs to.
// Every wait is bounded: past WAIT_POLLS polls the block sets the context's
// error word and returns without storing, and the host reports it
// (wait_status).  The others that wait look at the word too and give up with
// it, so that one limit's time is all that is lost; and what is enqueued behind
// a sort pass that gave up stores nothing: its input is not whole, and places
// taken from the counts of the true keys could lie outside the arrays.
#include "tk_emit.cuh"

#include <algorithm>

namespace tk {

constexpr uint64_t ST_PART = 1ULL << 62, ST_FULL = 2ULL << 62, ST_VALUE = (1ULL << 58) - 1;
constexpr uint32_t WAIT_POLLS = 1u << 20;   // of about a microsecond each
constexpr uint32_t WAIT_LOOK = 256;         // polls between two looks at the error word

__device__ __forceinline__ uint64_t st_read(const uint64_t *p) {
    return *reinterpret_cast<const volatile uint64_t *>(p);
}
__device__ __forceinline__ void st_write(uint64_t *p, uint64_t v) { *reinterpret_cast<volatile uint64_t *>(p) = v; }
__device__ __forceinline__ bool gave_up(const uint32_t *wait_err) {
    return *reinterpret_cast<const volatile uint32_t *>(wait_err) != 0;
}

// The polls a launch over `tiles` tiles may wait.  A test can have one such
// launch of a context leave out its first tile (*skip 1: the tickets start
// there, with a block fewer), so that every later tile's wait runs out.
static uint32_t wait_limit(tk_ctx *c, uint64_t tiles, uint32_t *skip) {
    *skip = 0;
    if (c->wait_test == 0 || tiles < 2 || --c->wait_test != 0) return WAIT_POLLS;
    *skip = 1;
    return c->wait_test_polls;
}

// ------------------------------------------------------------------ scan

constexpr int SN_THREADS = 256;
constexpr int SN_WARPS = SN_THREADS / 32;
constexpr int SN_ROUNDS = 4;                 // of four consecutive items per lane
constexpr uint64_t SN_TILE = (uint64_t)SN_THREADS * SN_ROUNDS * 4;

struct ScanHead {
    unsigned long long total;                // what the caller reads back, with err
    unsigned int err, ticket;
};

template <typename P>
__device__ __forceinline__ void load4(const uint32_t *in, P (&x)[4]) {
    const uint4 v = __ldg(reinterpret_cast<const uint4 *>(in));
    x[0] = v.x; x[1] = v.y; x[2] = v.z; x[3] = v.w;
}
__device__ __forceinline__ void load4(const uint64_t *in, uint64_t (&x)[4]) {
    const ulonglong2 a = __ldg(reinterpret_cast<const ulonglong2 *>(in)), b = __ldg(reinterpret_cast<const ulonglong2 *>(in) + 1);
    x[0] = a.x; x[1] = a.y; x[2] = b.x; x[3] = b.y;
}

// what the scan adds up for an input item, and the type that holds a tile's sum
struct ItemItself {
    using Part = uint64_t;
    __device__ __forceinline__ uint64_t operator()(uint64_t x) const { return x; }
};
struct RecordLength {   // ">COUNT\nKMER\n"
    using Part = uint32_t;
    int k;
    __device__ __forceinline__ uint32_t operator()(uint32_t count) const { return 3u + dec_digits(count) + (uint32_t)k; }
};

// A warp owns 512 consecutive items, four rounds of four per lane (16-byte
// loads and stores of consecutive lanes adjoin).  Bound by memory: 12 bytes
// an item for u32 input.  The three-kernel scan this replaces (reduce, one
// block over the tile sums, and a pass whose threads each walked 16
// consecutive items) took 10.5 us of kernels for 12,000 items and 45 us for 17M,
// and read its input twice.  With EVERY > 1 only every EVERY-th item's sum is
// stored, at out[i / EVERY].
template <typename Tin, typename F, int EVERY>
__global__ void __launch_bounds__(SN_THREADS) k_scan(F f, const Tin *__restrict__ in, uint64_t *__restrict__ out, uint64_t n,
                                                    int vec, ScanHead *__restrict__ head, uint64_t *__restrict__ state,
                                                    uint64_t *__restrict__ total_at, uint32_t *__restrict__ err_at,
                                                    uint32_t max_polls) {
    __shared__ uint64_t s_warp[SN_WARPS], s_before;
    __shared__ uint32_t s_tile, s_fail;
    if (threadIdx.x == 0) {
        s_tile = atomicAdd(&head->ticket, 1u);
        s_fail = 0;
    }
    __syncthreads();
    const uint64_t tile = s_tile;
    const unsigned lane = lane_id(), warp = threadIdx.x >> 5;
    const uint64_t first = tile * SN_TILE + (uint64_t)warp * (SN_TILE / SN_WARPS) + lane * 4;
    using P = typename F::Part;
    P x[SN_ROUNDS][4], pre[SN_ROUNDS], run = 0;
#pragma unroll
    for (int r = 0; r < SN_ROUNDS; r++) {
        const uint64_t i = first + (uint64_t)r * 128;
        if (vec && i + 4 <= n) {
            load4(in + i, x[r]);
        } else {
#pragma unroll
            for (int j = 0; j < 4; j++) x[r][j] = i + j < n ? (P)in[i + j] : 0;
        }
#pragma unroll
        for (int j = 0; j < 4; j++)
            if (i + j < n) x[r][j] = f(x[r][j]);
    }
#pragma unroll
    for (int r = 0; r < SN_ROUNDS; r++) {
        const P s = x[r][0] + x[r][1] + x[r][2] + x[r][3];
        const P inc = warp_incl_scan(s);
        pre[r] = run + inc - s;
        run += __shfl_sync(0xffffffffu, inc, 31);
    }
    if (lane == 0) s_warp[warp] = run;
    __syncthreads();
    if (warp == 0) {
        const uint64_t w = lane < SN_WARPS ? s_warp[lane] : 0;
        const uint64_t wi = warp_incl_scan(w);
        const uint64_t sum = __shfl_sync(0xffffffffu, wi, 31);
        if (lane < SN_WARPS) s_warp[lane] = wi - w;
        if (lane == 0) st_write(&state[tile], (tile ? ST_PART : ST_FULL) | sum);
        // 32 earlier tiles at a time, nearest first
        uint64_t before = 0;
        bool fail = false;
        for (int64_t t = (int64_t)tile - 1; t >= 0; t -= 32) {
            const int64_t mine = t - (int64_t)lane;
            uint64_t v = mine >= 0 ? 0 : ST_FULL;
            for (uint32_t polls = 0; __any_sync(0xffffffffu, v < ST_PART); polls++) {
                if (v < ST_PART) v = st_read(&state[mine]);
                fail = polls > max_polls || (polls % WAIT_LOOK == WAIT_LOOK - 1 && __any_sync(0xffffffffu, gave_up(err_at)));
                if (fail) break;   // uniform over the warp
            }
            const unsigned full = __ballot_sync(0xffffffffu, v >= ST_FULL);
            const int stop = full ? __ffs((int)full) - 1 : 31;
            before += warp_sum((int)lane <= stop ? (v & ST_VALUE) : 0ULL);
            if (full || fail) break;
        }
        if (lane == 0) {
            if (fail) {
                atomicExch(&head->err, 1u);
                atomicExch(err_at, 1u);
                s_fail = 1;
            } else {
                if (tile) st_write(&state[tile], ST_FULL | (before + sum));
                if (tile == (n - 1) / SN_TILE) {
                    head->total = before + sum;
                    if (total_at) *total_at = before + sum;
                }
            }
            s_before = before;
        }
    }
    __syncthreads();
    if (s_fail) return;
    const uint64_t base = s_before + s_warp[warp];
#pragma unroll
    for (int r = 0; r < SN_ROUNDS; r++) {
        const uint64_t i = first + (uint64_t)r * 128;
        uint64_t o[4];
        o[0] = base + pre[r];
#pragma unroll
        for (int j = 1; j < 4; j++) o[j] = o[j - 1] + x[r][j - 1];
        if (EVERY > 1) {
            static_assert(EVERY == 1 || EVERY % 4 == 0, "a lane's first item of four");
            if (i < n && i % EVERY == 0) out[i / EVERY] = o[0];
        } else if (vec && i + 4 <= n) {
            ulonglong2 *q = reinterpret_cast<ulonglong2 *>(out + i);
            q[0] = make_ulonglong2(o[0], o[1]);
            q[1] = make_ulonglong2(o[2], o[3]);
        } else {
#pragma unroll
            for (int j = 0; j < 4; j++)
                if (i + j < n) out[i + j] = o[j];
        }
    }
}

// Whether the wait limit of a sort or scan enqueued earlier ran out (each
// copies the context's error word to its page-locked word; call after a
// synchronisation).
int wait_status(tk_ctx *c) {
    if (!c->h_wait_err || *reinterpret_cast<volatile uint32_t *>(c->h_wait_err) == 0) return TK_OK;
    *c->h_wait_err = 0;
    cudaMemsetAsync(c->d_err + DE_COUNT, 0, 4, c->stream);
    return set_err(c, TK_E_CUDA, "sort or scan: the wait for an earlier tile ran out");
}

// The scan enqueued, its head left in *mem (the caller frees it).
template <typename Tin, int EVERY, typename F>
static int scan_enqueue(tk_ctx *c, F f, const Tin *in, uint64_t *out, uint64_t n, uint64_t *total_at, ScanHead **mem) {
    const uint64_t nt = (n + SN_TILE - 1) / SN_TILE;
    const size_t bytes = sizeof(ScanHead) + nt * 8;
    TK_TRY(dmalloc(c, (void **)mem, bytes, "scan tiles"));
    int e = cuda_check(c, cudaMemsetAsync(*mem, 0, bytes, c->stream), "scan reset");
    uint32_t skip;
    const uint32_t polls = wait_limit(c, nt, &skip);
    if (!e && skip) e = cuda_check(c, cudaMemsetAsync(&(*mem)->ticket, 1, 1, c->stream), "scan ticket");
    if (!e) {
        const int vec = (((uintptr_t)in | (EVERY > 1 ? 0 : (uintptr_t)out)) & 15u) == 0;
        k_scan<Tin, F, EVERY><<<(unsigned)nt - skip, SN_THREADS, 0, c->stream>>>(
            f, in, out, n, vec, *mem, reinterpret_cast<uint64_t *>(*mem + 1), total_at, c->d_err + DE_COUNT, polls);
        c->launches++;
        e = check_launch(c, "scan");
    }
    return e;
}

template <typename Tin, int EVERY = 1, typename F>
static int scan_impl(tk_ctx *c, F f, const Tin *in, uint64_t *out, uint64_t n, uint64_t *total_host) {
    *total_host = 0;
    if (n == 0) return TK_OK;
    ScanHead *head = nullptr, h;
    int e = scan_enqueue<Tin, EVERY>(c, f, in, out, n, nullptr, &head);
    if (!e) e = cuda_check(c, cudaMemcpyAsync(&h, head, sizeof h, cudaMemcpyDeviceToHost, c->stream), "scan total");
    if (!e) e = cuda_check(c, cudaStreamSynchronize(c->stream), "scan total sync");
    if (head) dfree(c, head);
    if (e) return e;
    if (h.err) {
        *c->h_wait_err = 0;
        cudaMemsetAsync(c->d_err + DE_COUNT, 0, 4, c->stream);
        return set_err(c, TK_E_CUDA, "scan: the wait for an earlier tile ran out");
    }
    TK_TRY(wait_status(c));
    *total_host = h.total;
    return TK_OK;
}

int scan_excl_u32_to_u64_async(tk_ctx *c, const uint32_t *in, uint64_t *out, uint64_t n, uint64_t *d_total) {
    if (n == 0) return cuda_check(c, cudaMemsetAsync(d_total, 0, 8, c->stream), "scan total");
    ScanHead *head = nullptr;
    int e = scan_enqueue<uint32_t, 1>(c, ItemItself{}, in, out, n, d_total, &head);
    if (!e) e = cuda_check(c, cudaMemcpyAsync(c->h_wait_err, c->d_err + DE_COUNT, 4, cudaMemcpyDeviceToHost, c->stream),
                           "scan status");
    if (head) dfree(c, head);
    return e;
}

int scan_excl_u64(tk_ctx *c, const uint64_t *in, uint64_t *out, uint64_t n, uint64_t *total_host) {
    return scan_impl<uint64_t>(c, ItemItself{}, in, out, n, total_host);
}

int scan_excl_u32_to_u64(tk_ctx *c, const uint32_t *in, uint64_t *out, uint64_t n, uint64_t *total_host) {
    return scan_impl<uint32_t>(c, ItemItself{}, in, out, n, total_host);
}

// Offsets of the dump records of n counts (k-mers of k bases).
int scan_record_lengths(tk_ctx *c, const uint32_t *counts, uint64_t *out, uint64_t n, int k, uint64_t *total_host) {
    return scan_impl<uint32_t, DUMP_BLOCK>(c, RecordLength{k}, counts, out, n, total_host);
}

// ------------------------------------------------------------------ radix sort

constexpr int RS_BITS = 8;
constexpr int RS_BINS = 1 << RS_BITS;
constexpr int RS_PASSES = 64 / RS_BITS;
constexpr int RC_THREADS = RS_BINS;          // the counting kernel: one digit per thread at its end

// One sort's device scratch, zeroed beforehand: the digit counts of every
// pass (turned into the digits' first places by the last counting block), the
// tile tickets, and the words the tiles of a pass publish, one per digit
// (each carries its pass, so one zeroing serves all passes).
struct SortHead {
    unsigned long long count[RS_PASSES][RS_BINS];
    unsigned int ticket[RS_PASSES];
    unsigned int done;
};

// The digit counts of all passes in one read of the keys.
__global__ void __launch_bounds__(RC_THREADS) k_rs_count(const uint64_t *__restrict__ keys, uint64_t n, int first_bit,
                                                        int passes, SortHead *__restrict__ head) {
    __shared__ uint32_t h[RS_PASSES][RS_BINS];
    __shared__ uint32_t s_last;
    __shared__ uint64_t sm[RC_THREADS / 32 + 1];
    for (int p = 0; p < passes; p++) h[p][threadIdx.x] = 0;
    __syncthreads();
    const uint64_t stride = (uint64_t)gridDim.x * RC_THREADS;
    for (uint64_t i0 = (uint64_t)blockIdx.x * RC_THREADS + threadIdx.x; i0 < n; i0 += 4 * stride) {
        uint64_t k[4];
#pragma unroll
        for (int u = 0; u < 4; u++) k[u] = i0 + u * stride < n ? keys[i0 + u * stride] >> first_bit : 0;
#pragma unroll
        for (int u = 0; u < 4; u++) {
            if (i0 + u * stride >= n) break;
            for (int p = 0; p < passes; p++) atomicAdd(&h[p][(k[u] >> (p * RS_BITS)) & (RS_BINS - 1)], 1u);
        }
    }
    __syncthreads();
    for (int p = 0; p < passes; p++) {
        const uint32_t v = h[p][threadIdx.x];
        if (v) atomicAdd(&head->count[p][threadIdx.x], (unsigned long long)v);
    }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) s_last = atomicAdd(&head->done, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    for (int p = 0; p < passes; p++) {
        const uint64_t v = __ldcg(&head->count[p][threadIdx.x]);
        uint64_t tot;
        const uint64_t ex = block_excl_scan<uint64_t>(v, sm, &tot);
        head->count[p][threadIdx.x] = ex;
    }
}

// One pass: a stable scatter of the pairs by one digit.  The tile's keys and
// values come into shared memory with cp.async (no registers in flight, so
// 36 warps per SM fit).  Warp w ranks its consecutive items in rounds of 32
// (eight ballots find the lanes with the same digit; the warp's running count
// per digit is in shared memory), a scan over (digit, warp) gives every item
// its place in the digit-sorted tile, thread d walks back over the earlier
// tiles' counts of digit d, LOOK words per step, and the tile leaves as one
// run per digit, consecutive threads storing consecutive items.  A last tile
// is filled up with keys of all ones, which rank behind its own pairs.
//
// Bound by the ranking's instructions and the tile's shared-memory gathers
// (ALU 56%, L1 59% of peak): 3.0 TB/s at 24 bytes a pair and pass.  Seven
// passes over 50 bits: 22M pairs 1.34 ms (2.05 before, with a histogram, a
// scan and a scatter kernel per pass), 140M 8.0, 30,000 0.076 (distinct keys take
// five, see k_sort_runs).  Tiles of 3840
// pairs (384 threads, three blocks per SM) from 1024 pairs per SM on (300,000
// pairs: 0.096 against 0.102 ms); below that tiles of 1024, whose shorter
// work is what counts (30,000 pairs: 0.076 against 0.089).  512 x 8, 512 x 12,
// 256 x 16, 256 x 24 and 384 x 16 lie within 5% at 140M pairs; match.any for
// the ranking takes 57 cycles of its pipe per round (1.87 ms at 22M), and
// keys held in registers leave 24 warps per SM (1.53).
constexpr int LOOK = 4;
template <int THREADS, int ITEMS>
struct SortTile {
    uint64_t key[THREADS * ITEMS];
    uint64_t gbase[RS_BINS];                 // digit d's run goes to [gbase[d] + its place in the tile, ...)
    uint32_t val[THREADS * ITEMS];
    uint32_t dstart[RS_BINS];
    uint16_t from[THREADS * ITEMS];          // place in the digit-sorted tile -> item
    uint16_t wcnt[THREADS / 32][RS_BINS];
};

template <int BYTES>
__device__ __forceinline__ void copy_async(void *smem, const void *gmem) {
    const uint32_t s = (uint32_t)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(s), "l"(gmem), "n"(BYTES) : "memory");
}

template <int THREADS, int ITEMS>
__global__ void __launch_bounds__(THREADS, THREADS == 384 ? 3 : 4)
    k_rs_pass(const uint64_t *__restrict__ keys, const uint32_t *__restrict__ vals, uint64_t *__restrict__ okeys,
              uint32_t *__restrict__ ovals, uint64_t n, int shift, int pass, SortHead *__restrict__ head,
              uint64_t *__restrict__ state, uint32_t *__restrict__ wait_err, uint32_t max_polls) {
    constexpr uint32_t TILE = THREADS * ITEMS;
    static_assert(THREADS >= RS_BINS && TILE <= 65536, "one digit per thread, 16-bit places");
    extern __shared__ __align__(16) unsigned char rs_mem[];
    SortTile<THREADS, ITEMS> &sm = *reinterpret_cast<SortTile<THREADS, ITEMS> *>(rs_mem);
    __shared__ uint32_t s_warp[RS_BINS / 32];
    __shared__ uint32_t s_tile, s_fail;
    if (threadIdx.x == 0) {
        s_fail = gave_up(wait_err);
        s_tile = atomicAdd(&head->ticket[pass], 1u);
    }
    for (uint32_t i = threadIdx.x; i < THREADS / 32 * RS_BINS / 2; i += THREADS)
        reinterpret_cast<uint32_t *>(&sm.wcnt[0][0])[i] = 0;
    __syncthreads();
    if (s_fail) return;   // an earlier pass or tile gave up
    const uint64_t tile = s_tile, t0 = tile * TILE;
    const uint32_t m = n - t0 < (uint64_t)TILE ? (uint32_t)(n - t0) : TILE;
    const unsigned lane = lane_id(), warp = threadIdx.x >> 5;
    const uint32_t first = warp * (32 * ITEMS) + lane;   // this lane's items: first, first + 32, ...
    const uint64_t *gk = keys + t0 + first;
    const uint32_t *gv = vals + t0 + first;
    if (m == TILE) {
#pragma unroll
        for (int r = 0; r < ITEMS; r++) copy_async<8>(&sm.key[first + r * 32], gk + r * 32);
        asm volatile("cp.async.commit_group;" ::: "memory");
#pragma unroll
        for (int r = 0; r < ITEMS; r++) copy_async<4>(&sm.val[first + r * 32], gv + r * 32);
    } else {
        for (int r = 0; r < ITEMS; r++) {
            if (first + r * 32 < m) copy_async<8>(&sm.key[first + r * 32], gk + r * 32);
            else sm.key[first + r * 32] = ~0ULL;
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
        for (int r = 0; r < ITEMS; r++)
            if (first + r * 32 < m) copy_async<4>(&sm.val[first + r * 32], gv + r * 32);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    const unsigned lt_mask = (1u << lane) - 1u;
    uint16_t *mycnt = sm.wcnt[warp];
    uint32_t pos[ITEMS];   // (digit << 16) | rank among the warp's items of that digit
#pragma unroll
    for (int r = 0; r < ITEMS; r++) {
        const uint32_t d = (uint32_t)(sm.key[first + r * 32] >> shift) & (RS_BINS - 1);   // its own copy
        unsigned peers = ~0u;
#pragma unroll
        for (int b = 0; b < RS_BITS; b++) {
            const unsigned ones = __ballot_sync(0xffffffffu, (d >> b) & 1u);
            peers &= (d >> b) & 1u ? ones : ~ones;
        }
        const int leader = __ffs((int)peers) - 1;
        uint32_t cur = 0;
        if ((int)lane == leader) {
            cur = mycnt[d];
            mycnt[d] = (uint16_t)(cur + __popc(peers));
        }
        __syncwarp();
        pos[r] = (d << 16) + __shfl_sync(0xffffffffu, cur, leader) + __popc(peers & lt_mask);
    }
    __syncthreads();
    // thread d: digit d's count in each warp, turned into the counts of the warps before
    const bool digit = THREADS == RS_BINS || threadIdx.x < RS_BINS;
    const uint64_t tag = (uint64_t)(pass + 1) << 58;
    uint64_t *words = state + threadIdx.x;   // used by the digits' threads only
    uint32_t mine = 0;
    if (digit) {
#pragma unroll
        for (int w = 0; w < THREADS / 32; w++) {
            const uint32_t x = sm.wcnt[w][threadIdx.x];
            sm.wcnt[w][threadIdx.x] = (uint16_t)mine;
            mine += x;
        }
        st_write(words + tile * RS_BINS, (tile ? ST_PART : ST_FULL) | tag | mine);
    }
    // the digits' first places in the tile: a scan over the first RS_BINS threads
    uint32_t at = 0;
    if (digit) {
        at = warp_incl_scan(mine);
        if (lane == 31) s_warp[warp] = at;
        at -= mine;
    }
    __syncthreads();
    if (digit) {
        for (unsigned w = 0; w < warp; w++) at += s_warp[w];
        sm.dstart[threadIdx.x] = at;
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < ITEMS; r++) {
        const uint32_t d = pos[r] >> 16;
        sm.from[(pos[r] & 0xFFFFu) + sm.dstart[d] + mycnt[d]] = (uint16_t)(first + r * 32);
    }
    if (digit) {
        // digit d's pairs in the earlier tiles
        uint64_t before = 0;
        bool found = tile == 0;
        const uint64_t *q = words + tile * RS_BINS;   // the words of the tile last taken
        for (uint32_t polls = 0; !found && polls <= max_polls; polls++) {
            if (polls % WAIT_LOOK == WAIT_LOOK - 1 && gave_up(wait_err)) break;
            uint64_t w[LOOK];
#pragma unroll
            for (int i = 0; i < LOOK; i++) {
                const uint64_t *x = q - (i + 1) * RS_BINS;
                w[i] = x >= state ? st_read(x) : 0;
            }
#pragma unroll
            for (int i = 0; i < LOOK; i++) {
                // a word of this pass, next in line: taken; else the rest is read again
                if (found || ((uint32_t)(w[i] >> 58) & 15u) != (uint32_t)(pass + 1)) break;
                before += w[i] & ST_VALUE;
                found = w[i] >= ST_FULL;
                q -= RS_BINS;
            }
        }
        if (!found) {
            atomicExch(wait_err, 1u);
            s_fail = 1;
        } else if (tile) {
            st_write(words + tile * RS_BINS, ST_FULL | tag | (before + mine));
        }
        sm.gbase[threadIdx.x] = head->count[pass][threadIdx.x] + before - at;
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    if (s_fail) return;
    auto put = [&](uint32_t i) {
        const uint32_t f = sm.from[i];
        const uint64_t key = sm.key[f];
        const uint64_t o = sm.gbase[(uint32_t)(key >> shift) & (RS_BINS - 1)] + i;
        okeys[o] = key;
        ovals[o] = sm.val[f];
    };
    if (m == TILE) {
#pragma unroll
        for (int r = 0; r < ITEMS; r++) put(r * THREADS + threadIdx.x);
    } else {
        for (uint32_t i = threadIdx.x; i < m; i += THREADS) put(i);
    }
}

template <int THREADS, int ITEMS>
static int sort_run(tk_ctx *c, uint64_t *ka, uint32_t *va, uint64_t *kb, uint32_t *vb, uint64_t n, int passes,
                    int first_bit) {
    const uint64_t tile = (uint64_t)THREADS * ITEMS, nt = (n + tile - 1) / tile;
    constexpr int smem = (int)sizeof(SortTile<THREADS, ITEMS>);
    unsigned char *mem = nullptr;
    const size_t head_bytes = (sizeof(SortHead) + 255) / 256 * 256, bytes = head_bytes + nt * RS_BINS * 8;
    TK_TRY(dmalloc(c, (void **)&mem, bytes, "radix sort tiles"));
    SortHead *head = reinterpret_cast<SortHead *>(mem);
    uint64_t *state = reinterpret_cast<uint64_t *>(mem + head_bytes);
    int e = cuda_check(c, cudaMemsetAsync(mem, 0, bytes, c->stream), "radix sort reset");
    if (!e) e = cuda_check(c, cudaFuncSetAttribute(k_rs_pass<THREADS, ITEMS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                   smem), "radix sort smem");
    if (!e) {
        const uint64_t want = (n + 4 * RC_THREADS - 1) / (4 * RC_THREADS);
        k_rs_count<<<(unsigned)std::min<uint64_t>(want, (uint64_t)c->sm_count * 8), RC_THREADS, 0, c->stream>>>(
            ka, n, first_bit, passes, head);
        c->launches++;
        for (int p = 0; p < passes; p++) {
            uint32_t skip;
            const uint32_t polls = wait_limit(c, nt, &skip);
            if (skip) cudaMemsetAsync(&head->ticket[p], 1, 1, c->stream);
            k_rs_pass<THREADS, ITEMS><<<(unsigned)nt - skip, THREADS, smem, c->stream>>>(
                ka, va, kb, vb, n, first_bit + p * RS_BITS, p, head, state, c->d_err + DE_COUNT, polls);
            c->launches++;
            std::swap(ka, kb);
            std::swap(va, vb);
        }
        e = check_launch(c, "radix sort");
    }
    if (!e) e = cuda_check(c, cudaMemcpyAsync(c->h_wait_err, c->d_err + DE_COUNT, 4, cudaMemcpyDeviceToHost, c->stream),
                           "radix sort status");
    dfree(c, mem);
    return e;
}

// Sorts by key bits [first_bit, first_bit + bits), 8 bits per pass; stable.
// An overrun wait is reported by the next scan, or by wait_status after a
// synchronisation.
int radix_sort_pairs(tk_ctx *c, uint64_t *keys, uint32_t *vals, uint64_t n, int bits, uint64_t *tmp_keys,
                     uint32_t *tmp_vals, bool *result_in_tmp, int first_bit) {
    *result_in_tmp = false;
    if (n <= 1 || bits <= 0) return TK_OK;
    const int passes = (std::min(bits, 64 - first_bit) + RS_BITS - 1) / RS_BITS;
    *result_in_tmp = passes & 1;
    if (n >= (uint64_t)c->sm_count * 1024)
        return sort_run<384, 10>(c, keys, vals, tmp_keys, tmp_vals, n, passes, first_bit);
    return sort_run<256, 4>(c, keys, vals, tmp_keys, tmp_vals, n, passes, first_bit);
}

// ---- the last bits of a sort of distinct keys.  With the pairs in order of all
// but their r <= 10 lowest bits, the keys that agree in the rest form runs of at
// most 2^r, short ones mostly (k-mers that differ in their last bases), and every
// run is put in order in place.  A thread ranks its key among the keys of its
// run, FX_NEAR or fewer, by comparing; a longer run is ranked by its block
// through a bitmap of its lowest bits (the keys are distinct).  A run belongs to
// the block that holds its first pair; a block that reads a neighbour's run while
// that is reordered sees only its upper bits, which are the same in every order.
// Bound by instructions (issue slots 81% busy): 22M pairs 92 us, 39M 194 us, where
// the two passes it saves of seven over 50 bits took 355 and 618 (counting with
// five digits takes 59 us for 68): 1.31 -> 1.05 ms for the sort of 22M. 10 bits, so
// that 25-mers save two passes and a run fits one block with four keys a thread.
constexpr int FX_THREADS = 256, FX_ITEMS = 4, FX_TILE = FX_THREADS * FX_ITEMS;
constexpr int FX_NEAR = 64;
constexpr int FX_BITS = 10;

__global__ void __launch_bounds__(FX_THREADS) k_sort_runs(uint64_t *keys, uint32_t *vals, uint64_t n, int r,
                                                          const uint32_t *__restrict__ wait_err) {
    if (*wait_err) return;   // a pass gave up: the pairs are not in order
    static_assert(FX_TILE >= (1 << FX_BITS) && FX_THREADS >= FX_NEAR, "a run fits a block");
    __shared__ uint64_t s[FX_TILE + FX_NEAR + 1];   // the pair before the tile, the tile, FX_NEAR pairs behind it
    __shared__ uint32_t s_long[FX_TILE / FX_NEAR + 1], n_long, map[1 << (FX_BITS - 5)], below[1 << (FX_BITS - 5)];
    const uint64_t t0 = (uint64_t)blockIdx.x * FX_TILE;
    const int tid = (int)threadIdx.x;
    const int from = t0 ? 0 : 1;                                                      // valid places: [from, end)
    const int end = 1 + (int)min(n - t0, (uint64_t)(FX_TILE + FX_NEAR));
    if (tid == 0) n_long = 0;
    for (int j = from + tid; j < end; j += FX_THREADS) s[j] = keys[t0 + j - 1];
    __syncthreads();
    int to[FX_ITEMS + 1];
    uint32_t val[FX_ITEMS + 1];
#pragma unroll
    for (int u = 0; u <= FX_ITEMS; u++) {
        to[u] = -1;
        const int j = 1 + u * FX_THREADS + tid;   // (the last round: the pairs behind the tile)
        if (j >= end || j > FX_TILE + FX_NEAR) continue;
        const uint64_t key = s[j], top = key >> r;
        const bool prev = j > from && s[j - 1] >> r == top, next = j + 1 < end && s[j + 1] >> r == top;
        if (!prev && !next) continue;
        int a = j, less = 0;
        while (a > from && j - a <= FX_NEAR && s[a - 1] >> r == top) less += s[--a] < key;
        if (a == 0 || a > FX_TILE || j - a > FX_NEAR) continue;   // another block's run, or a long one
        int b = j + 1;
        while (b < end && b - a <= FX_NEAR && s[b] >> r == top) less += s[b++] < key;
        if (b - a > FX_NEAR) {
            if (a == j) s_long[atomicAdd(&n_long, 1u)] = (uint32_t)j;
            continue;
        }
        if (a + less != j) {
            to[u] = a + less;
            val[u] = vals[t0 + j - 1];
        }
    }
    __syncthreads();
#pragma unroll
    for (int u = 0; u <= FX_ITEMS; u++) {
        if (to[u] < 0) continue;
        keys[t0 + to[u] - 1] = s[1 + u * FX_THREADS + tid];
        vals[t0 + to[u] - 1] = val[u];
    }
    for (uint32_t q = 0; q < n_long; q++) {
        const uint64_t g0 = t0 + s_long[q] - 1, top = s[s_long[q]] >> r;
        uint64_t key[FX_ITEMS];
        bool in[FX_ITEMS];
        for (int i = tid; i < 1 << (FX_BITS - 5); i += FX_THREADS) map[i] = 0;
        __syncthreads();
#pragma unroll
        for (int u = 0; u < FX_ITEMS; u++) {
            const uint64_t g = g0 + u * FX_THREADS + tid;
            in[u] = false;
            if (g >= n) continue;
            key[u] = keys[g];
            in[u] = key[u] >> r == top;
            if (!in[u]) continue;
            val[u] = vals[g];
            const uint32_t low = (uint32_t)key[u] & ((1u << r) - 1u);
            atomicOr(&map[low >> 5], 1u << (low & 31u));
        }
        __syncthreads();
        if (tid < 32) {
            const uint32_t c = __popc(map[tid]);
            below[tid] = warp_incl_scan(c) - c;
        }
        __syncthreads();
#pragma unroll
        for (int u = 0; u < FX_ITEMS; u++) {
            if (!in[u]) continue;
            const uint32_t low = (uint32_t)key[u] & ((1u << r) - 1u);
            const uint64_t g = g0 + below[low >> 5] + __popc(map[low >> 5] & ((1u << (low & 31u)) - 1u));
            keys[g] = key[u];
            vals[g] = val[u];
        }
        __syncthreads();
    }
}

// Sorts pairs of distinct keys by their lowest `bits` bits (the others are 0):
// 8-bit passes over the upper bits and k_sort_runs for up to FX_BITS lowest ones.
int sort_distinct_pairs(tk_ctx *c, uint64_t *keys, uint32_t *vals, uint64_t n, int bits, uint64_t *tmp_keys,
                        uint32_t *tmp_vals, bool *result_in_tmp) {
    const int passes = std::max(1, (bits - FX_BITS + 7) / 8), low = std::max(0, bits - 8 * passes);
    TK_TRY(radix_sort_pairs(c, keys, vals, n, bits - low, tmp_keys, tmp_vals, result_in_tmp, low));
    if (low == 0 || n <= 1) return TK_OK;
    k_sort_runs<<<(unsigned)((n + FX_TILE - 1) / FX_TILE), FX_THREADS, 0, c->stream>>>(
        *result_in_tmp ? tmp_keys : keys, *result_in_tmp ? tmp_vals : vals, n, low, c->d_err + DE_COUNT);
    c->launches++;
    return check_launch(c, "sort runs");
}

}  // namespace tk
