// tk_dbg.cu -- per-record de Bruijn k-mer graphs of the Inchworm bundle
// (Inchworm FastaToDeBruijn --fasta bundled_iworm_contigs.fasta -K 24
// --graph_per_record, called at Trinity:2298-2302; its output is cut into one
// file per component by util/support_scripts/partition_chrysalis_graphs_n_reads.pl).
//
// Per bundle record (one component: its Inchworm contigs joined by 'X'), the
// distinct (K+1)-mers in order of first occurrence, each with the node of the
// window just before its first occurrence (-1 at a contig start or a break)
// and its number of occurrences in the record (a k-mer and its reverse
// complement are one node unless strand-specific).  Text: "Component <id>"
// then "<node>\t<prev>\t<count>\t<kmer>" per node; a record without any
// window is left out.
//
// GPU plan, all over the record-concatenated bundle read set, a thread per
// window end position throughout:
//  1. every record gets a slice of a hash table (a power of two, at least 1.5
//     times its bases); each window is inserted into its record's slice, which
//     keeps its count and the first position it ends at, and the position
//     keeps the slot;
//  2. a position is a node when its slot's first position is its own: a bit per
//     position, and the nodes in the 32 positions of every word scanned;
//     node id = nodes before the position - nodes before the record;
//  3. prev through the slot of the window before; line lengths, a scan, and one
//     thread per line writing it.
// Neighbouring threads work on neighbouring positions, so the slices in use at
// any time are those of a short stretch of the bundle and stay in L2.  (Three
// radix sorts -- by k-mer, by record, by first position -- and the passes that
// joined their results took 3.0 of the 4.5 ms of 30,000 contigs.)
#include "tk_emit.cuh"
#include "tk_warp.cuh"

#include <algorithm>
#include <vector>

namespace tk {

constexpr uint32_t NO_NODE = 0xFFFFFFFFu;

__device__ __forceinline__ uint32_t dbg_dec_len(uint64_t v) {
    uint32_t n = 1;
    while (v >= 10) {
        v /= 10;
        n++;
    }
    return n;
}

__device__ __forceinline__ char *dbg_put_dec(char *o, uint64_t v) {
    const uint32_t n = dbg_dec_len(v);
    for (uint32_t i = n; i > 0; i--) {
        o[i - 1] = (char)('0' + v % 10);
        v /= 10;
    }
    return o + n;
}

constexpr int DBG_THREADS = 256;

// A block takes DBG_STEPS stretches of DBG_THREADS positions, one after
// another; the record of its first position is searched once, and every thread
// walks on from the record of its last position.  (13.6M positions, insert /
// heads / lines with one stretch per block 0.41 / 0.18 / 0.25 ms: the search's
// dependent loads.)
constexpr int DBG_STEPS = 8;
constexpr uint64_t DBG_SPAN = (uint64_t)DBG_THREADS * DBG_STEPS;

// the record holding position p, the block's first
__device__ __forceinline__ uint32_t dbg_record(const uint64_t *__restrict__ rd_off, uint64_t n_rec, uint64_t p) {
    __shared__ uint32_t s_rec;
    if (threadIdx.x == 0) {
        uint64_t lo = 0, hi = n_rec;   // the largest r with rd_off[r] <= p
        while (hi - lo > 1) {
            const uint64_t mid = (lo + hi) >> 1;
            if (rd_off[mid] <= p) lo = mid;
            else hi = mid;
        }
        s_rec = (uint32_t)lo;
    }
    __syncthreads();
    return s_rec;
}

// Calls f(e, r) for every position of this thread in the block's stretches (e
// past the last position included, so that a warp stays together) and the
// record r holding it.
template <typename F>
__device__ __forceinline__ void dbg_positions(const uint64_t *__restrict__ rd_off, uint64_t n_rec, F &&f) {
    const uint64_t p0 = (uint64_t)blockIdx.x * DBG_SPAN;
    uint32_t r = dbg_record(rd_off, n_rec, p0);
    uint64_t next = __ldg(rd_off + r + 1);
    for (int st = 0; st < DBG_STEPS; st++) {
        const uint64_t e = p0 + (uint64_t)st * DBG_THREADS + threadIdx.x;
        while (e >= next && r + 1 < n_rec) next = __ldg(rd_off + ++r + 1);
        f(e, r);
    }
}

// 1. slots of each record's slice
__global__ void k_dbg_slices(const uint64_t *__restrict__ rd_off, uint64_t n_rec, uint64_t *__restrict__ size) {
    const uint64_t r = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= n_rec) return;
    const uint64_t bases = rd_off[r + 1] - rd_off[r] - 1;
    uint64_t s = 32;
    while (2 * s < 3 * bases) s <<= 1;
    size[r] = s;
}

template <bool CANON>
__global__ void __launch_bounds__(DBG_THREADS) k_dbg_insert(const uint64_t *__restrict__ codes,
                                                            const uint32_t *__restrict__ inv, uint64_t n_pos, int k1,
                                                            const uint64_t *__restrict__ rd_off, uint64_t n_rec,
                                                            const uint64_t *__restrict__ base,
                                                            const uint64_t *__restrict__ size, Slot *__restrict__ slots,
                                                            uint32_t *__restrict__ slot_of) {
    const uint64_t inner = (1ULL << (2 * k1 - 2)) - 1;
    dbg_positions(rd_off, n_rec, [&](uint64_t e, uint32_t r) {
        if (e >= n_pos) return;
        uint64_t key;
        if (!window_at<CANON>(codes, inv, e, k1, key)) {
            slot_of[e] = NO_NODE;
            return;
        }
        Slot *t = slots + base[r];
        const uint32_t mask = (uint32_t)(size[r] - 1);
        // the slot of the key, added `times` times from position e on (the slice has room for every window of its record)
        auto insert = [&](uint32_t times) {
            const uint64_t mine = e << 32 | times;   // first position, count
            for (uint32_t s = (uint32_t)mix64(key) & mask;; s = (s + 1) & mask) {
                if (s == NO_NODE) continue;   // no position can name that slot
                const ulonglong2 was = slot_claim(t + s, 0, key, mine);
                if (was.x == EMPTY_KEY) return s;
                if (was.x == key) {
                    atomicAdd(&t[s].val, times);
                    if ((uint32_t)(was.y >> 32) > (uint32_t)e) atomicMin(&t[s].pad, (uint32_t)e);
                    return s;
                }
            }
        };
        uint32_t s = NO_NODE;
        if (((key ^ key >> 2) & inner) == 0) {
            // a stretch of one letter is one k-mer: its windows in the warp go in together
            // (3 Mb of A one by one 6.3 ms, atomics on one slot; 0.5 this way)
            const unsigned here = __activemask();
            const unsigned alike = __match_any_sync(here, key) & __match_any_sync(here, r);
            const int lead = __ffs((int)alike) - 1;   // the first position
            if ((int)lane_id() == lead) s = insert((uint32_t)__popc(alike));
            s = __shfl_sync(alike, s, lead);
        } else {
            s = insert(1);
        }
        slot_of[e] = s;
    });
}

// 2. a bit per position (bit i of word j: position 32j + i) that is a node, and the nodes of each word
__global__ void __launch_bounds__(DBG_THREADS) k_dbg_heads(uint64_t n_pos, const uint64_t *__restrict__ rd_off,
                                                           uint64_t n_rec, const uint64_t *__restrict__ base,
                                                           const Slot *__restrict__ slots,
                                                           const uint32_t *__restrict__ slot_of,
                                                           uint32_t *__restrict__ head, uint32_t *__restrict__ heads) {
    dbg_positions(rd_off, n_rec, [&](uint64_t e, uint32_t r) {
        const uint32_t s = e < n_pos ? slot_of[e] : NO_NODE;
        const bool node = s != NO_NODE && slots[base[r] + s].pad == (uint32_t)e;
        __syncwarp();
        const uint32_t bits = __ballot_sync(0xffffffffu, node);
        if (lane_id() == 0 && e < n_pos) {
            head[e >> 5] = bits;
            heads[e >> 5] = __popc(bits);
        }
    });
}

// the nodes ending before position e
__device__ __forceinline__ uint32_t dbg_rank(const uint32_t *__restrict__ head, const uint64_t *__restrict__ before,
                                             uint64_t e) {
    return (uint32_t)before[e >> 5] + __popc(head[e >> 5] & ((1u << (e & 31)) - 1u));
}

struct DbgLine {
    uint32_t id;       // node id in its record
    int32_t prev;      // -1: none
    uint32_t count;
    uint32_t rec;      // record index; header line before the record's first node
};

// 3. every node's line (in position order), its window's first position and its text length
__global__ void __launch_bounds__(DBG_THREADS) k_dbg_lines(uint64_t n_pos, const uint64_t *__restrict__ rd_off,
                                                           uint64_t n_rec, const uint64_t *__restrict__ base,
                                                           const Slot *__restrict__ slots,
                                                           const uint32_t *__restrict__ slot_of,
                                                           const uint32_t *__restrict__ head,
                                                           const uint64_t *__restrict__ before,
                                                           const uint64_t *__restrict__ comp, int k1,
                                                           DbgLine *__restrict__ line, uint64_t *__restrict__ first,
                                                           uint32_t *__restrict__ len,
                                                           unsigned long long *__restrict__ n_comp) {
    dbg_positions(rd_off, n_rec, [&](uint64_t e, uint32_t r) {
        if (e >= n_pos || !((head[e >> 5] >> (e & 31)) & 1u)) return;
        const Slot *t = slots + base[r];
        const uint32_t j = dbg_rank(head, before, e), r0 = dbg_rank(head, before, rd_off[r]);
        DbgLine L;
        L.id = j - r0;
        L.count = t[slot_of[e]].val;
        L.rec = r;
        // the window just before the first occurrence, when it is a valid window
        // (it then lies in the same contig of the same record)
        const uint32_t ps = e > 0 ? slot_of[e - 1] : NO_NODE;
        L.prev = ps == NO_NODE ? -1 : (int32_t)(dbg_rank(head, before, t[ps].pad) - r0);
        line[j] = L;
        first[j] = e - (uint64_t)k1 + 1;
        uint32_t n = dec_digits(L.id) + 1 + (L.prev < 0 ? 2 : dec_digits((uint32_t)L.prev)) + 1 + dec_digits(L.count) + 1 +
                     (uint32_t)k1 + 1;
        if (L.id == 0) {
            n += 10 + dbg_dec_len(comp[r]) + 1;   // "Component " id "\n"
            atomicAdd(n_comp, 1ULL);
        }
        len[j] = n;
    });
}

// 4. one thread per node line, formatted in the block's shared-memory buffer
// and stored in aligned 16-byte pieces (13.6M lines, 490 MB: a thread storing
// its line's bytes one by one took 2.24 ms).  The k-mer comes from the codes: a
// window holds A/C/G/T only, in upper case in the read array.
constexpr int DBG_LINE = 10 + 1 + 11 + 1 + 10 + 1 + MAX_K + 1;
constexpr int DBG_BYTES = (DBG_THREADS * (DBG_LINE + 10 + 20 + 1) + 16 + 15) & ~15;

__global__ void __launch_bounds__(DBG_THREADS) k_dbg_write(const DbgLine *__restrict__ line,
                                                           const uint64_t *__restrict__ first,
                                                           const uint64_t *__restrict__ off, uint64_t n_nodes,
                                                           uint64_t total, const uint64_t *__restrict__ comp,
                                                           const uint64_t *__restrict__ codes, int k1,
                                                           char *__restrict__ out) {
    __shared__ __align__(16) char buf[DBG_BYTES];
    const uint64_t j0 = (uint64_t)blockIdx.x * DBG_THREADS, j = j0 + threadIdx.x;
    const uint64_t w0 = off[j0], w1 = j0 + DBG_THREADS < n_nodes ? off[j0 + DBG_THREADS] : total;
    if (j < n_nodes) {
        const DbgLine L = line[j];
        char *o = buf + (w0 & 15) + (off[j] - w0);
        if (L.id == 0) {
            const char hdr[] = "Component ";
            for (int i = 0; i < 10; i++) o[i] = hdr[i];
            o = dbg_put_dec(o + 10, comp[L.rec]);
            *o++ = '\n';
        }
        o = put_dec(o, L.id, dec_digits(L.id));
        *o++ = '\t';
        if (L.prev < 0) {
            *o++ = '-';
            *o++ = '1';
        } else {
            o = put_dec(o, (uint32_t)L.prev, dec_digits((uint32_t)L.prev));
        }
        *o++ = '\t';
        o = put_dec(o, L.count, dec_digits(L.count));
        *o++ = '\t';
        const uint64_t p = first[j], q = p >> 5;
        const int s = 2 * (int)(p & 31);
        const uint64_t hi = __ldg(codes + q);
        const uint64_t w = s ? (hi << s) | (__ldg(codes + q + 1) >> (64 - s)) : hi;   // 32 positions from p on
        put_kmer_line(o, w >> (64 - 2 * k1), k1);
    }
    __syncthreads();
    block_store(buf, out, w0, (uint32_t)(w1 - w0));
}

static unsigned dbg_grid(uint64_t n, int threads) { return (unsigned)std::max<uint64_t>(1, (n + threads - 1) / threads); }

// Device allocations released on every path out of dbg_build.
struct DbgScratch {
    tk_ctx *c;
    std::vector<void *> p;
    explicit DbgScratch(tk_ctx *ctx) : c(ctx) {}
    int get(void **out, uint64_t bytes, const char *what) {
        int e = dmalloc(c, out, bytes ? bytes : 8, what);
        if (!e) p.push_back(*out);
        return e;
    }
    ~DbgScratch() {
        for (void *q : p) dfree(c, q);
    }
};

int component_ids(tk_ctx *c, const tk_reads *b, uint64_t *d_ids);

int dbg_build(tk_dbg *g, const tk_reads *b) {
    tk_ctx *c = g->ctx;
    const int k1 = g->k + 1;
    const uint64_t n_rec = b->n_reads, n_pos = b->seq_len;
    g->n_nodes = 0;
    g->n_components = 0;
    g->text_len = 0;
    if (n_rec == 0 || n_pos < (uint64_t)k1) return TK_OK;
    DbgScratch sc(c);
    cudaEvent_t ev;
    prof_begin(c, TK_KID_DBG, &ev);
    if (n_pos >= NO_NODE) return set_err(c, TK_E_RANGE, "FastaToDeBruijn: a bundle of 2^32 - 1 bytes or more");
    const uint64_t n_words = (n_pos + 31) / 32;
    uint32_t *slot_of = nullptr, *head = nullptr, *heads = nullptr;
    uint64_t *size = nullptr, *base = nullptr, *before = nullptr, n_slots = 0, G = 0;
    Slot *slots = nullptr;
    TK_TRY(sc.get((void **)&size, n_rec * 8, "slice sizes"));
    TK_TRY(sc.get((void **)&base, n_rec * 8, "slice starts"));
    k_dbg_slices<<<dbg_grid(n_rec, 256), 256, 0, c->stream>>>(b->d_rd_off, n_rec, size);
    c->launches++;
    TK_TRY(scan_excl_u64(c, size, base, n_rec, &n_slots));
    TK_TRY(sc.get((void **)&slots, n_slots * sizeof(Slot), "k-mer slices"));
    TK_TRY(sc.get((void **)&slot_of, n_pos * 4, "window slots"));
    TK_TRY(sc.get((void **)&head, n_words * 4, "node bits"));
    TK_TRY(sc.get((void **)&heads, n_words * 4, "nodes per word"));
    TK_TRY(sc.get((void **)&before, n_words * 8, "nodes before"));
    table_fill_empty(c, slots, n_slots, 0);
    const unsigned grid = (unsigned)((n_pos + DBG_SPAN - 1) / DBG_SPAN);
    if (g->strand)
        k_dbg_insert<false><<<grid, DBG_THREADS, 0, c->stream>>>(b->d_codes, b->d_inv, n_pos, k1, b->d_rd_off, n_rec, base,
                                                                 size, slots, slot_of);
    else
        k_dbg_insert<true><<<grid, DBG_THREADS, 0, c->stream>>>(b->d_codes, b->d_inv, n_pos, k1, b->d_rd_off, n_rec, base,
                                                                size, slots, slot_of);
    k_dbg_heads<<<grid, DBG_THREADS, 0, c->stream>>>(n_pos, b->d_rd_off, n_rec, base, slots, slot_of, head, heads);
    c->launches += 2;
    TK_TRY(check_launch(c, "de Bruijn windows"));
    TK_TRY(scan_excl_u32_to_u64(c, heads, before, n_words, &G));
    if (G == 0) {
        prof_end(c, TK_KID_DBG, ev, 0);
        return TK_OK;
    }
    uint64_t *d_comp = nullptr, *ofirst = nullptr, *loff = nullptr;
    uint32_t *len = nullptr;
    unsigned long long *d_ncomp = nullptr;
    DbgLine *line = nullptr;
    TK_TRY(sc.get((void **)&d_ncomp, 8, "component count"));
    TK_CUDA(c, cudaMemsetAsync(d_ncomp, 0, 8, c->stream));
    TK_TRY(sc.get((void **)&d_comp, n_rec * 8, "component ids"));
    TK_TRY(sc.get((void **)&ofirst, G * 8, "node first positions"));
    TK_TRY(sc.get((void **)&line, G * sizeof(DbgLine), "node lines"));
    TK_TRY(sc.get((void **)&len, G * 4, "line lengths"));
    TK_TRY(sc.get((void **)&loff, (G + 1) * 8, "line offsets"));
    TK_TRY(component_ids(c, b, d_comp));
    k_dbg_lines<<<grid, DBG_THREADS, 0, c->stream>>>(n_pos, b->d_rd_off, n_rec, base, slots, slot_of, head, before, d_comp,
                                                     k1, line, ofirst, len, d_ncomp);
    c->launches++;
    TK_TRY(check_launch(c, "de Bruijn lines"));
    uint64_t total = 0;
    TK_TRY(scan_excl_u32_to_u64(c, len, loff, G, &total));
    char *text = nullptr;
    TK_TRY(dmalloc(c, (void **)&text, total + 1, "de Bruijn text"));
    k_dbg_write<<<dbg_grid(G, DBG_THREADS), DBG_THREADS, 0, c->stream>>>(line, ofirst, loff, G, total, d_comp, b->d_codes, k1, text);
    c->launches++;
    int e = check_launch(c, "de Bruijn text");
    if (e) {
        dfree(c, text);
        return e;
    }
    unsigned long long n_comp = 0;
    e = cuda_check(c, cudaMemcpyAsync(&n_comp, d_ncomp, 8, cudaMemcpyDeviceToHost, c->stream), "component count");
    if (!e) e = cuda_check(c, cudaStreamSynchronize(c->stream), "de Bruijn sync");
    if (e) {
        dfree(c, text);
        return e;
    }
    prof_end(c, TK_KID_DBG, ev, n_pos);
    g->d_text = text;
    g->text_len = total;
    g->n_nodes = G;
    g->n_components = n_comp;
    return TK_OK;
}

}  // namespace tk
