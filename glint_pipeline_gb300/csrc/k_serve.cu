/*
 * k_serve.cu -- contact-trace queries over the flushed store, served with
 * continuous batching.
 *
 * Reference: id_search_in_CTB / id_search_in_disk (tracing/workbench.cpp:
 * 397-444) read one object's keys per call: its sid picks a CTF (or the
 * oversize buffer, sid 1), CTF::binary_search / oversize_buffer::
 * search_buffer find its first key and the walk of search_SSTable visits the
 * rest (tracing/step_merge.cpp:67-115, 501-568); the targets of one hop are
 * the search list of the next (search_multi_pid, tracing/process.cpp:476-495).
 *
 * Device form: every query owns a slot: a bitmap of the objects it has reached
 * and one of those the current hop reaches.  One launch advances every active
 * slot by one hop: its items are (slot, frontier object, kept block) triples,
 * over the kept blocks whose time span can meet the slot's window; the
 * object's sid, first and count in the block locate its keys, which are
 * decoded as CTF::parse_key does (tracing/step_merge.cpp:335-345), and each
 * target inside the time window that the slot has not reached is marked.  A
 * scan over the slots' marks then lists them, ascending, slot after slot: that
 * list is the hop's result and the next hop's frontiers.  Between launches the
 * host retires finished queries and admits waiting ones into free slots
 * (continuous batching); a slot's result only depends on its own query.
 *
 * Bound: the hop's dependent reads, and around it launches and copies.  With
 * each new object appended to its slot's list by an atomic, the lists then
 * radix-sorted by (slot, id), 10 separate copies of control arrays and a
 * synchronisation of its own for the seeds, a 2-hop query from 1000 seeds over
 * 16 blocks of 3M objects took 97 operations on the stream (820 us); marks, the
 * scan and one control copy take 13 (225 us, 184 of them the two hops).
 */
#include <algorithm>
#include <cstring>
#include <deque>
#include <unordered_map>
#include <vector>

#include "scan.cuh"
#include "serve_queue.h"
#include "store_codec.cuh"

namespace glint {

struct SlotParam {
    uint32_t t_start, t_end, window, pad;
};

struct HopArgs {
    const StoreBlockDev *blocks;
    uint32_t N;
    uint32_t words;                        /* bitmap words per slot, a multiple of a scan thread's items */
    uint32_t *visited;                     /* [slot][words] reached so far */
    uint32_t *fresh;                       /* [slot][words] reached by this hop */
    const SlotParam *param;                /* [slot] */
    unsigned long long *scanned;           /* [slot] keys read */
    const uint32_t *active;                /* [A] slots taking part in this launch */
    const uint32_t *front;                 /* [A] their frontier sizes */
    const uint32_t *const *front_ids;      /* [A] their frontiers */
    const unsigned long long *prefix;      /* [A + 1] their items (frontier x blocks), prefix sums */
    const uint32_t *rel;                   /* each active slot's blocks, concatenated */
    const uint32_t *rel_off;               /* [A + 1] where each active slot's blocks start in rel */
    uint32_t A;
};

/* the reached-set word of target for slot s (all ones past N) */
__device__ inline uint32_t visited_word(const HopArgs &a, uint32_t s, uint32_t target) {
    return target < a.N ? __ldcg(&a.visited[(size_t)s * a.words + (target >> 5)]) : ~0u;
}

/* marks target reached by this hop for slot s, given its reached-set word
 * `seen` (visited_word).  A query's bits only go from 0 to 1, so a set bit
 * read from L2 is final and saves the atomic; a clear one is settled by it. */
__device__ inline void visit_seen(const HopArgs &a, uint32_t s, uint32_t target, uint32_t seen) {
    if (target >= a.N) return;
    const uint32_t bit = 1u << (target & 31);
    const size_t w = (size_t)s * a.words + (target >> 5);
    if (!(seen & bit) && !(atomicOr(&a.visited[w], bit) & bit)) atomicOr(&a.fresh[w], bit);
}

/* one item's keys as the hop reads them: where they start, how many, and
 * how a key decodes (kind 1: the oversize buffer's 16-byte keys; kind 2: a
 * CTF's packed keys, whose end, duration and target fields lie in the 64
 * bits from byte off of the key when fast is set) */
struct HopItem {
    const uint8_t *base;
    const uint8_t *end;      /* the end of the block's packed keys */
    uint32_t n, s, kind, pad;
    uint32_t kb, off, fast, mbr_bit;
    uint32_t end_bit, dur_bit, end_mask, dur_mask;
    uint32_t id_mask, etm, window, t_start;
    uint32_t t_end, pad0, pad1, pad2;
};

constexpr int kHopThreads = 256;
constexpr int kHopKeys = 4; /* keys per lane per round */

/* the 64 bits at p, which need not be aligned; whole words while they stay
 * inside the buffer ending at `end` (whose start is 8-aligned) */
__device__ inline unsigned long long load_u64(const uint8_t *p, const uint8_t *end) {
    const uintptr_t a = (uintptr_t)p;
    const uint64_t *w = (const uint64_t *)(a & ~(uintptr_t)7);
    const uint32_t sh = (uint32_t)(a & 7) * 8;
    if ((const uint8_t *)(w + 2) <= end) {
        const uint64_t lo = w[0];
        return sh ? (lo >> sh) | (w[1] << (64 - sh)) : lo;
    }
    unsigned long long v = 0;
    for (uint32_t i = 0; i < 8 && p + i < end; ++i) v |= (unsigned long long)p[i] << (8 * i);
    return v;
}

/* Each warp takes 32 consecutive items, one per lane, and looks up the
 * object's sid, first key and key count in the item's block.  An object has
 * anywhere from none to hundreds of keys in a block, so the warp then walks
 * the keys of all 32 items together, 32 at a time: lane l takes the warp's
 * key k0 + l, finds its item by a binary search over the items' key counts'
 * prefix sums, and reads that item's decoding from shared memory.  Every lane
 * has a key on every round but the last, and the warp's loop count is its
 * total keys / 32 instead of its largest item's key count.  A lane decodes
 * kHopKeys keys before it reads their bitmap words, so that their loads
 * overlap. */
__global__ void __launch_bounds__(kHopThreads) k_serve_hop(HopArgs a) {
    __shared__ HopItem items[kHopThreads];
    __shared__ uint32_t koff[kHopThreads];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    HopItem *wi = items + wib * 32;
    uint32_t *wo = koff + wib * 32;
    const unsigned long long total = a.prefix[a.A];
    const unsigned long long warps = (unsigned long long)gridDim.x * (kHopThreads / 32);
    for (unsigned long long w = blockIdx.x * (unsigned long long)(kHopThreads / 32) + wib; w * 32 < total;
         w += warps) {
        const unsigned long long it = w * 32 + lane;
        HopItem h;
        h.n = 0;
        h.kind = 0;
        h.s = 0;
        if (it < total) {
            uint32_t lo = 0, hi = a.A; /* prefix[lo] <= it < prefix[lo + 1] */
            while (hi - lo > 1) {
                const uint32_t mid = (lo + hi) / 2;
                if (a.prefix[mid] <= it) lo = mid;
                else hi = mid;
            }
            /* block-major within a slot: consecutive items take consecutive
             * frontier objects (ascending ids) of one block, whose sids,
             * key ranges and keys then lie close together */
            const uint32_t fr = a.front[lo];
            const unsigned long long local = it - a.prefix[lo];
            uint32_t bi, f;
            if (local < (1ull << 32)) {
                bi = (uint32_t)local / fr;
                f = (uint32_t)local - bi * fr;
            } else {
                bi = (uint32_t)(local / fr);
                f = (uint32_t)(local - (unsigned long long)bi * fr);
            }
            const uint32_t b = a.rel[a.rel_off[lo] + bi];
            const uint32_t s = a.active[lo];
            const SlotParam sp = a.param[s];
            const uint32_t obj = a.front_ids[lo][f];
            const StoreBlockDev &blk = a.blocks[b];
            const uint32_t sid = blk.sids[obj];
            h.s = s;
            h.window = sp.window;
            h.t_start = sp.t_start;
            h.t_end = sp.t_end;
            h.etm = blk.end_time_min;
            if (sid == 1) {
                h.n = blk.count[obj];
                h.kind = 1;
                h.base = reinterpret_cast<const uint8_t *>(blk.okeys + blk.first[obj]);
            } else if (sid >= 2 && sid - 2 < blk.C) {
                const uint32_t c = sid - 2;
                const glint_ctf_meta &m = blk.ctfs[c];
                const uint32_t kb = m.key_bit / 8, mb = m.mbr_bit, eb = m.end_bit, db = m.duration_bit,
                               ib = m.id_bit;
                h.n = blk.count[obj];
                h.kind = 2;
                h.kb = kb;
                h.mbr_bit = mb;
                h.off = mb / 8;
                h.fast = (mb & 7) + eb + db + ib <= 64;
                h.end_bit = eb;
                h.dur_bit = db;
                h.end_mask = eb >= 32 ? 0xffffffffu : (1u << eb) - 1u;
                h.dur_mask = db >= 32 ? 0xffffffffu : (1u << db) - 1u;
                h.id_mask = ib >= 32 ? 0xffffffffu : (1u << ib) - 1u;
                h.end = blk.keys + blk.key_bytes;
                h.base = blk.keys + blk.byte_index[c] + (unsigned long long)(blk.first[obj] - blk.key_index[c]) * kb;
            }
        }
        /* keys read, per slot: the lanes of one slot add with one reduction */
        const unsigned withkeys = __ballot_sync(0xffffffffu, h.n != 0);
        if (h.n) {
            const unsigned peers = __match_any_sync(withkeys, h.s);
            const uint32_t grp = __reduce_add_sync(peers, h.n);
            if (lane == __ffs(peers) - 1) atomicAdd(&a.scanned[h.s], (unsigned long long)grp);
        }
        /* exclusive prefix of the key counts over the warp */
        uint32_t incl = h.n;
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += v;
        }
        const uint32_t T = __shfl_sync(0xffffffffu, incl, 31);
        wi[lane] = h;
        wo[lane] = incl - h.n;
        __syncwarp();
        /* kHopKeys keys per lane in flight: their loads, then their bitmap
         * words, then the (rare) atomics and appends */
        for (uint32_t k0 = 0; k0 < T; k0 += 32 * kHopKeys) {
            uint32_t tg[kHopKeys], sl[kHopKeys], seen[kHopKeys];
#pragma unroll
            for (int u = 0; u < kHopKeys; ++u) {
                const uint32_t k = k0 + u * 32 + lane;
                tg[u] = 0xffffffffu;
                sl[u] = 0;
                if (k < T) {
                    /* the last item whose first key is at or before k: it has
                     * keys, since an item without keys shares its offset with
                     * the item after it, and k < T rules out the last lane */
                    uint32_t lo = 0;
#pragma unroll
                    for (uint32_t step = 16; step; step >>= 1)
                        if (lo + step < 32 && wo[lo + step] <= k) lo += step;
                    const HopItem &x = wi[lo];
                    const uint32_t j = k - wo[lo];
                    sl[u] = x.s;
                    uint32_t end, duration, t;
                    if (x.kind == 2 && x.fast) {
                        /* end, duration and target from one 64-bit window */
                        unsigned long long v = load_u64(x.base + (size_t)j * x.kb + x.off, x.end);
                        v >>= x.mbr_bit & 7;
                        end = ((uint32_t)v & x.end_mask) + x.etm;
                        v >>= x.end_bit;
                        duration = (uint32_t)v & x.dur_mask;
                        v >>= x.dur_bit;
                        t = (uint32_t)v & x.id_mask;
                    } else if (x.kind == 2) {
                        unsigned __int128 v = load_key(x.base + (size_t)j * x.kb, x.kb, x.end);
                        v >>= x.mbr_bit;
                        end = (uint32_t)(v & ((1ull << x.end_bit) - 1)) + x.etm;
                        v >>= x.end_bit;
                        duration = (uint32_t)(v & ((1ull << x.dur_bit) - 1));
                        v >>= x.dur_bit;
                        t = (uint32_t)v & x.id_mask;
                    } else {
                        const ulonglong2 kk = reinterpret_cast<const ulonglong2 *>(x.base)[j];
                        end = (uint32_t)kk.x + x.etm;
                        duration = (uint32_t)(kk.x >> 32);
                        t = (uint32_t)kk.y & ((1u << 26) - 1);
                    }
                    const uint32_t start = end - duration;
                    if (!x.window || (start < x.t_end && x.t_start < end)) tg[u] = t;
                }
            }
#pragma unroll
            for (int u = 0; u < kHopKeys; ++u) seen[u] = visited_word(a, sl[u], tg[u]);
#pragma unroll
            for (int u = 0; u < kHopKeys; ++u) visit_seen(a, sl[u], tg[u], seen[u]);
        }
        __syncwarp();
    }
}

/* ---- pull hops -----------------------------------------------------------
 * When a slot's frontier is at least as large as the set of objects it has
 * not reached, the hop runs from the other side: every unreached object u
 * reads its own keys in the window's blocks and is reached when one of its
 * targets was reached before this hop.  A meeting's two keys (a -> b and
 * b -> a, cuda/geometry.cu:714-734) lie in the same block with the same
 * times, so u has a key to a reached object v exactly when v has one to u;
 * and v was reached at the previous hop, since a v reached earlier would have
 * reached u already.  The reached set is read as it stood before the hop
 * (its marks join it after it, MarkOut), so the hop's result is the one
 * the frontier's own walk gives, and u stops at its first such key. */

/* one warp per bitmap word: for each of its unreached objects, the object's
 * keys in the slot's blocks, 32 blocks at a time, until one reaches an object
 * reached before this hop */
__global__ void __launch_bounds__(256) k_serve_pull(HopArgs b) {
    const int lane = threadIdx.x & 31;
    const uint32_t nw = (b.N + 31) / 32;
    const unsigned long long total = (unsigned long long)b.A * nw;
    const unsigned long long nwarps = (unsigned long long)gridDim.x * (blockDim.x / 32);
    for (unsigned long long w = (blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x) / 32; w < total;
         w += nwarps) {
        const uint32_t lo = (uint32_t)(w / nw), word = (uint32_t)(w - (unsigned long long)lo * nw);
        const uint32_t s = b.active[lo];
        const uint32_t *vis = b.visited + (size_t)s * b.words;
        uint32_t left = ~vis[word];
        if (word == nw - 1 && (b.N & 31)) left &= (1u << (b.N & 31)) - 1u;
        if (!left) continue;
        const SlotParam sp = b.param[s];
        const uint32_t r0 = b.rel_off[lo], nrel = b.rel_off[lo + 1] - r0;
        uint32_t got = 0;
        unsigned long long keys = 0;
        for (; left; left &= left - 1) {
            const uint32_t u = word * 32 + (uint32_t)__ffs(left) - 1;
            bool found = false;
            for (uint32_t r = 0; r < nrel && !found; r += 32) {
                bool hit = false;
                if (r + lane < nrel) {
                    const StoreBlockDev &blk = b.blocks[b.rel[r0 + r + lane]];
                    const uint32_t sid = blk.sids[u];
                    uint32_t n = 0;
                    if (sid == 1) {
                        n = blk.count[u];
                        const ulonglong2 *k = blk.okeys + blk.first[u];
                        for (uint32_t j = 0; j < n && !hit; ++j) {
                            const ulonglong2 kk = k[j];
                            const uint32_t end = (uint32_t)kk.x + blk.end_time_min, dur = (uint32_t)(kk.x >> 32);
                            const uint32_t t = (uint32_t)kk.y & ((1u << 26) - 1);
                            ++keys;
                            if (sp.window && !((end - dur) < sp.t_end && sp.t_start < end)) continue;
                            if (t < b.N && ((vis[t >> 5] >> (t & 31)) & 1u)) hit = true;
                        }
                    } else if (sid >= 2 && sid - 2 < blk.C) {
                        const uint32_t c = sid - 2;
                        const glint_ctf_meta &m = blk.ctfs[c];
                        const uint32_t kb = m.key_bit / 8;
                        n = blk.count[u];
                        const uint8_t *base =
                            blk.keys + blk.byte_index[c] + (unsigned long long)(blk.first[u] - blk.key_index[c]) * kb;
                        const uint8_t *kend = blk.keys + blk.key_bytes;
                        for (uint32_t j = 0; j < n && !hit; ++j) {
                            unsigned __int128 v = load_key(base + (size_t)j * kb, kb, kend);
                            v >>= m.mbr_bit;
                            const uint32_t end = (uint32_t)(v & ((1ull << m.end_bit) - 1)) + blk.end_time_min;
                            v >>= m.end_bit;
                            const uint32_t dur = (uint32_t)(v & ((1ull << m.duration_bit) - 1));
                            v >>= m.duration_bit;
                            const uint32_t t = (uint32_t)(v & ((1ull << m.id_bit) - 1));
                            ++keys;
                            if (sp.window && !((end - dur) < sp.t_end && sp.t_start < end)) continue;
                            if (t < b.N && ((vis[t >> 5] >> (t & 31)) & 1u)) hit = true;
                        }
                    }
                }
                found = __any_sync(0xffffffffu, hit);
            }
            if (found) got |= 1u << (u & 31);
        }
        for (int o = 16; o > 0; o >>= 1) keys += __shfl_down_sync(0xffffffffu, keys, o);
        if (lane == 0) {
            if (keys) atomicAdd(&b.scanned[s], keys);
            if (got) b.fresh[(size_t)s * b.words + word] = got;
        }
    }
}

/* the start of a round: the reached sets of the slots just admitted (their
 * indices among the active ones come first in `admitted`) and the marks of
 * every active slot cleared */
__global__ void __launch_bounds__(256) k_serve_begin(HopArgs a, const uint32_t *__restrict__ admitted,
                                                     uint32_t n_admitted) {
    const unsigned long long per = a.words / 4, na = per * n_admitted, total = na + per * a.A;
    for (unsigned long long i = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; i < total;
         i += (unsigned long long)gridDim.x * blockDim.x) {
        const bool adm = i < na;
        const unsigned long long j = adm ? i : i - na;
        const uint32_t r = (uint32_t)(j / per);
        const uint32_t s = adm ? admitted[r] : a.active[r];
        uint4 *w = reinterpret_cast<uint4 *>((adm ? a.visited : a.fresh) + (size_t)s * a.words);
        w[j - (unsigned long long)r * per] = make_uint4(0, 0, 0, 0);
        if (adm && j == (unsigned long long)r * per) a.scanned[s] = 0;
    }
}

/* the seeds of newly admitted slots are reached */
__global__ void k_serve_seed(const uint32_t *__restrict__ seeds, const uint32_t *__restrict__ sprefix,
                             const uint32_t *__restrict__ slots, uint32_t n_slots, HopArgs a) {
    const uint32_t total = sprefix[n_slots];
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
        uint32_t lo = 0, hi = n_slots;
        while (hi - lo > 1) {
            const uint32_t mid = (lo + hi) / 2;
            if (sprefix[mid] <= i) lo = mid;
            else hi = mid;
        }
        const uint32_t p = seeds[i];
        atomicOr(&a.visited[(size_t)slots[lo] * a.words + (p >> 5)], 1u << (p & 31));
    }
}

/* the marks of the active slots, slot after slot, as one scan for each group of
 * slots whose objects a 32-bit sum counts (mark_group): each word's
 * count of marks, then its ids at its place of the result list; a slot's first
 * place is where its ids start.  Pull hops read the reached sets as they stood
 * before the hop, so their marks join them here (a walk's marks are in). */
struct MarkIn {
    const uint32_t *fresh;
    const uint32_t *active;
    uint32_t words;
    __device__ const uint32_t *word(uint32_t i) const {
        const uint32_t r = i / words;
        return fresh + (size_t)active[r] * words + (i - r * words);
    }
    __device__ uint32_t at(uint32_t i) const { return __popc(*word(i)); }
    __device__ void load(uint32_t base, uint32_t n, uint32_t (&v)[kScanItems]) const {
        /* n and words are multiples of kScanItems: a thread's words are of
         * one slot, and aligned */
#pragma unroll
        for (int k = 0; k < kScanItems; ++k) v[k] = 0;
        if (base >= n) return;
        const uint4 *w = reinterpret_cast<const uint4 *>(word(base));
#pragma unroll
        for (int k = 0; k < kScanItems; k += 4) {
            const uint4 x = w[k / 4];
            v[k] = __popc(x.x);
            v[k + 1] = __popc(x.y);
            v[k + 2] = __popc(x.z);
            v[k + 3] = __popc(x.w);
        }
    }
};
struct MarkOut {
    MarkIn in;
    uint32_t *visited;
    uint32_t *ids;             /* the result list */
    unsigned long long *off;   /* [A + 1] */
    uint32_t A;
    bool later;                /* off[0] holds the total of the groups of slots before this one */
    __device__ unsigned long long before() const { return later ? off[0] : 0ull; }
    __device__ void total(uint32_t, uint32_t sum) const { off[A] = before() + sum; }
    __device__ void store(uint32_t base, uint32_t n, const uint32_t (&v)[kScanItems],
                          const uint32_t (&o)[kScanItems]) const {
        if (base >= n) return;
        const uint32_t r = base / in.words, w0 = base - r * in.words;
        const unsigned long long b = before();
        if (w0 == 0 && !(later && r == 0)) off[r] = b + o[0];
        const uint32_t *f = in.word(base);
        uint32_t *vis = visited + (size_t)in.active[r] * in.words + w0;
#pragma unroll
        for (int k = 0; k < kScanItems; ++k) {
            if (!v[k]) continue;
            uint32_t m = f[k];
            unsigned long long at = b + o[k];
            vis[k] |= m;
            for (; m; m &= m - 1) ids[at++] = (w0 + k) * 32 + (uint32_t)__ffs(m) - 1;
        }
    }
};

} // namespace glint

using namespace glint;

struct glint_server {
    glint_ctx *ctx = nullptr;
    uint32_t slots = 0;
    uint32_t words = 0;
    uint32_t *visited = nullptr, *fresh = nullptr;
    uint32_t *ids[2] = {nullptr, nullptr}; /* the result lists of this round and the last: [slots * N] */
    uint32_t side = 0;                     /* which of them the next round writes */
    unsigned long long *out = nullptr;     /* keys read per slot [slots], the result list's offsets [slots + 1] */
    unsigned long long *h_out = nullptr;   /* page-locked: the same */
    uint8_t *ctl = nullptr, *h_ctl = nullptr; /* a round's control arrays: device, page-locked */
    uint64_t ctl_cap = 0;
    uint32_t *h_ids = nullptr;             /* page-locked: results on their way to the queries */
    void *scan_tmp = nullptr;
    uint64_t next_ticket = 1;
    std::deque<PendingQuery> queue;
    std::vector<SlotState> state;
    std::vector<SlotParam> hparam;
    std::unordered_map<uint64_t, FinishedQuery> done;
};

constexpr uint64_t kIdsStage = 1u << 20; /* ids per copy to the host */

static void server_release(glint_server *v) {
    void *ps[] = {v->visited, v->fresh, v->ids[0], v->ids[1], v->out, v->ctl, v->scan_tmp};
    for (void *p : ps)
        if (p) cudaFree(p);
    void *hs[] = {v->h_out, v->h_ctl, v->h_ids};
    for (void *p : hs)
        if (p) cudaFreeHost(p);
    v->visited = v->fresh = v->ids[0] = v->ids[1] = v->h_ids = nullptr;
    v->out = v->h_out = nullptr;
    v->ctl = v->h_ctl = nullptr;
    v->ctl_cap = 0;
    v->scan_tmp = nullptr;
}

/* a round's control arrays, laid out one after the other in page-locked
 * memory and copied to the device at once */
class Control {
public:
    template <class T>
    size_t add(const T *p, size_t n) {
        const size_t at = (bytes_.size() + 15) & ~(size_t)15;
        bytes_.resize(at + sizeof(T) * std::max<size_t>(n, 1));
        if (n) std::memcpy(bytes_.data() + at, p, sizeof(T) * n);
        return at;
    }
    template <class T>
    size_t add(const std::vector<T> &v) {
        return add(v.data(), v.size());
    }
    /* room for n bytes in v's buffers (grown by half again, kept) */
    static cudaError_t room(glint_server *v, size_t n) {
        if (v->ctl_cap >= n) return cudaSuccess;
        if (v->ctl) cudaFree(v->ctl);
        if (v->h_ctl) cudaFreeHost(v->h_ctl);
        v->ctl = v->h_ctl = nullptr;
        v->ctl_cap = 0;
        const size_t cap = std::max<size_t>(n + n / 2, 1u << 16);
        cudaError_t e = cudaMalloc((void **)&v->ctl, cap);
        if (e == cudaSuccess) e = cudaMallocHost((void **)&v->h_ctl, cap);
        if (e == cudaSuccess) v->ctl_cap = cap;
        return e;
    }
    size_t size() const { return bytes_.size(); }
    uint8_t *data() { return bytes_.data(); }

private:
    std::vector<uint8_t> bytes_;
};

extern "C" glint_status glint_server_create(glint_ctx *c, uint32_t max_slots, glint_server **out) {
    if (!c || !out || max_slots == 0) return GLINT_ERR_INVALID_ARGUMENT;
    *out = nullptr;
    cudaSetDevice(c->device);
    glint_server *v = new glint_server();
    v->ctx = c;
    static_assert(kScanItems == 8, "slot_words");
    v->words = slot_words(c->N);
    /* admission by memory: a slot costs its two bitmaps and its part of the
     * two result lists */
    const size_t slot_bytes = sizeof(uint32_t) * (2 * (size_t)v->words + 2 * (size_t)c->N) + 64;
    size_t free_b = 0, total_b = 0;
    cudaMemGetInfo(&free_b, &total_b);
    const size_t fit = (free_b / 2) / slot_bytes;
    v->slots = (uint32_t)std::min<size_t>(max_slots, std::max<size_t>(fit, 1));
    const uint32_t S = v->slots;
    cudaError_t e = cudaSuccess;
    auto A = [&](void **p, size_t n) {
        if (e == cudaSuccess) e = cudaMalloc(p, n ? n : 1);
    };
    const size_t scan_bytes = scan_tmp_bytes((size_t)v->words * std::min(S, mark_group(c->N)));
    A((void **)&v->visited, sizeof(uint32_t) * (size_t)v->words * S);
    A((void **)&v->fresh, sizeof(uint32_t) * (size_t)v->words * S);
    A((void **)&v->ids[0], sizeof(uint32_t) * (size_t)c->N * S);
    A((void **)&v->ids[1], sizeof(uint32_t) * (size_t)c->N * S);
    A((void **)&v->out, sizeof(unsigned long long) * (2 * (size_t)S + 1));
    A(&v->scan_tmp, scan_bytes);
    if (e == cudaSuccess) e = cudaMallocHost((void **)&v->h_out, sizeof(unsigned long long) * (2 * (size_t)S + 1));
    if (e == cudaSuccess) e = cudaMallocHost((void **)&v->h_ids, sizeof(uint32_t) * kIdsStage);
    if (e == cudaSuccess) e = Control::room(v, 1u << 16);
    if (e == cudaSuccess) e = cudaMemsetAsync(v->scan_tmp, 0, scan_bytes, c->stream);
    if (e != cudaSuccess) {
        server_release(v);
        delete v;
        c->last_error = std::string("server: ") + cudaGetErrorString(e);
        return e == cudaErrorMemoryAllocation ? GLINT_ERR_OUT_OF_MEMORY : GLINT_ERR_CUDA;
    }
    v->state.resize(S);
    v->hparam.resize(S);
    c->servers.push_back(v);
    *out = v;
    return GLINT_OK;
}

/* a server whose context was destroyed first is detached: its device memory
 * is released with the context and only the handle remains */
extern "C" glint_status glint_server_destroy(glint_server *v) {
    if (!v) return GLINT_OK;
    if (v->ctx) {
        glint_ctx *c = v->ctx;
        cudaSetDevice(c->device);
        cudaStreamSynchronize(c->stream);
        server_release(v);
        c->servers.erase(std::remove(c->servers.begin(), c->servers.end(), v), c->servers.end());
        if (c->server == v) c->server = nullptr;
    }
    delete v;
    return GLINT_OK;
}

extern "C" uint32_t glint_server_slots(const glint_server *v) { return v ? v->slots : 0u; }

extern "C" glint_status glint_server_submit(glint_server *v, const glint_query *q, uint64_t *ticket) {
    if (v && !v->ctx) return GLINT_ERR_STATE;
    if (!v || !q || (q->n_seeds && !q->seeds) || q->hops == 0 || q->hops > kMaxHops) return GLINT_ERR_INVALID_ARGUMENT;
    PendingQuery p;
    p.ticket = v->next_ticket++;
    p.seeds.assign(q->seeds, q->seeds + q->n_seeds);
    p.hops = q->hops;
    p.t_start = q->t_start;
    p.t_end = q->t_end;
    v->queue.push_back(std::move(p));
    if (ticket) *ticket = v->queue.back().ticket;
    return GLINT_OK;
}

static glint_status server_fail(glint_server *v, cudaError_t e, const char *where) {
    v->ctx->last_error = std::string("server ") + where + ": " + cudaGetErrorString(e);
    cudaGetLastError(); /* a refused allocation is this call's error, not the next launch's */
    return e == cudaErrorMemoryAllocation ? GLINT_ERR_OUT_OF_MEMORY : GLINT_ERR_CUDA;
}

/* the slot's query is done */
static void server_finish(glint_server *v, SlotState &st, uint64_t keys_scanned) {
    for (uint32_t h = st.hop; h < kMaxHops; ++h) st.hop_end[h] = st.ids.size();
    FinishedQuery f;
    f.ids = std::move(st.ids);
    std::memcpy(f.hop_end, st.hop_end, sizeof(f.hop_end));
    f.keys_scanned = keys_scanned;
    v->done[st.ticket] = std::move(f);
    st = SlotState();
}

extern "C" glint_status glint_server_step(glint_server *v, uint32_t *n_active, uint32_t *n_queued) {
    if (!v) return GLINT_ERR_INVALID_ARGUMENT;
    if (!v->ctx) return GLINT_ERR_STATE;
    glint_ctx *c = v->ctx;
    cudaSetDevice(c->device);
    cudaStream_t s = c->stream;
    const uint32_t N = c->N;
    cudaError_t e;
    Control ctl;
    /* the kept blocks, as device descriptors */
    const uint32_t nb = (uint32_t)c->ctbs.size();
    std::vector<StoreBlockDev> bd(nb);
    for (uint32_t i = 0; i < nb; ++i) {
        const StoreBlock &b = c->ctbs[i];
        bd[i] = StoreBlockDev{b.keys, b.key_bytes, b.ctfs, b.key_index, b.byte_index, b.sids, b.first, b.count,
                              b.okeys, b.end_time_min, b.C};
    }
    const size_t at_blocks = ctl.add(bd);

    /* undone at every return before the round's launches have run */
    Admission adm(v->queue, v->state);
    adm.take(N);
    const std::vector<uint32_t> &admitted = adm.slots, &seeds = adm.seeds, &sprefix = adm.sprefix;
    for (size_t i = 0; i < admitted.size(); ++i) {
        const PendingQuery &q = adm.query(i);
        v->hparam[admitted[i]] = SlotParam{q.t_start, q.t_end, (q.t_start == 0 && q.t_end == 0) ? 0u : 1u, 0u};
    }
    const size_t at_seeds = ctl.add(seeds), at_sprefix = ctl.add(sprefix), at_admitted = ctl.add(admitted);

    /* one hop for every active slot, over the kept blocks that can hold a
     * key inside its window: a key of a block ends at most at end_time_max
     * and starts no earlier than start_min, and it counts when
     * start < t_end and t_start < end.  Frontier walks first, then the pull
     * slots (their frontier reaches at least as many objects as are left). */
    std::vector<uint32_t> act, rel, front, rel_off(1, 0);
    std::vector<unsigned long long> prefix(1, 0);
    uint32_t n_push = 0;
    for (int pass = 0; pass < 2; ++pass)
        for (uint32_t k = 0; k < v->slots; ++k) {
            const SlotState &st = v->state[k];
            if (!st.busy || st.hop >= st.hops) continue;
            const bool pull = (uint64_t)st.frontier >= (uint64_t)N - st.reached;
            if (pull != (pass == 1)) continue;
            act.push_back(k);
            front.push_back(st.frontier);
            const SlotParam &sp = v->hparam[k];
            uint32_t nrel = 0;
            for (uint32_t i = 0; i < nb; ++i) {
                const StoreBlock &b = c->ctbs[i];
                if (sp.window && b.spans_known && !(b.start_min < sp.t_end && sp.t_start < b.end_time_max)) continue;
                rel.push_back(i);
                ++nrel;
            }
            rel_off.push_back((uint32_t)rel.size());
            if (!pull) {
                prefix.push_back(prefix.back() + (unsigned long long)st.frontier * nrel);
                ++n_push;
            }
        }
    if (!act.empty()) {
        const uint32_t A = (uint32_t)act.size();
        const size_t at_param = ctl.add(v->hparam), at_act = ctl.add(act), at_front = ctl.add(front),
                     at_prefix = ctl.add(prefix), at_rel = ctl.add(rel), at_rel_off = ctl.add(rel_off);
        std::vector<const uint32_t *> fids(A, nullptr);
        const size_t at_fids = ctl.add(fids);
        if ((e = Control::room(v, ctl.size())) != cudaSuccess) return server_fail(v, e, "control arrays");
        for (uint32_t i = 0; i < admitted.size(); ++i)
            v->state[admitted[i]].front_ids = reinterpret_cast<const uint32_t *>(v->ctl + at_seeds) + sprefix[i];
        for (uint32_t i = 0; i < A; ++i) fids[i] = v->state[act[i]].front_ids;
        std::memcpy(ctl.data() + at_fids, fids.data(), sizeof(uint32_t *) * A);
        std::memcpy(v->h_ctl, ctl.data(), ctl.size());
        cudaMemcpyAsync(v->ctl, v->h_ctl, ctl.size(), cudaMemcpyHostToDevice, s);
        auto dev = [&](auto *type, size_t at) { return reinterpret_cast<decltype(type)>(v->ctl + at); };
        HopArgs a;
        a.blocks = dev((const StoreBlockDev *)nullptr, at_blocks);
        a.N = N;
        a.words = v->words;
        a.visited = v->visited;
        a.fresh = v->fresh;
        a.param = dev((const SlotParam *)nullptr, at_param);
        a.scanned = v->out;
        a.active = dev((const uint32_t *)nullptr, at_act);
        a.front = dev((const uint32_t *)nullptr, at_front);
        a.front_ids = dev((const uint32_t *const *)nullptr, at_fids);
        a.prefix = dev((const unsigned long long *)nullptr, at_prefix);
        a.rel = dev((const uint32_t *)nullptr, at_rel);
        a.rel_off = dev((const uint32_t *)nullptr, at_rel_off);
        a.A = A;
        const uint32_t n_adm = (uint32_t)admitted.size();
        const uint32_t *d_adm = dev((const uint32_t *)nullptr, at_admitted);
        k_serve_begin<<<grid_for((uint64_t)(v->words / 4) * (A + n_adm), 256, 152u * 8u), 256, 0, s>>>(a, d_adm, n_adm);
        if (!seeds.empty())
            k_serve_seed<<<grid_for(seeds.size(), 256), 256, 0, s>>>(dev((const uint32_t *)nullptr, at_seeds),
                                                                     dev((const uint32_t *)nullptr, at_sprefix), d_adm,
                                                                     n_adm, a);
        const unsigned long long items = prefix.back();
        if (items) {
            a.A = n_push;
            k_serve_hop<<<grid_for((items + 31) / 32, kHopThreads / 32, 152u * 8u), kHopThreads, 0, s>>>(a);
        }
        if (A > n_push) {
            HopArgs b = a;
            b.active = a.active + n_push;
            b.rel_off = a.rel_off + n_push;
            b.A = A - n_push;
            k_serve_pull<<<grid_for((uint64_t)b.A * ((N + 31) / 32), 8, 152u * 16u), 256, 0, s>>>(b);
        }
        MarkOut mo;
        mo.visited = v->visited;
        mo.ids = v->ids[v->side];
        const uint32_t group = mark_group(N);
        for (uint32_t r = 0; r < A; r += group) {
            mo.in = MarkIn{v->fresh, a.active + r, v->words};
            mo.off = v->out + v->slots + r;
            mo.A = std::min(group, A - r);
            mo.later = r != 0;
            scan_launch(mo.in, mo, v->words * mo.A, nullptr, v->scan_tmp, s);
        }
        cudaMemcpyAsync(v->h_out, v->out, sizeof(unsigned long long) * (v->slots + (size_t)A + 1),
                        cudaMemcpyDeviceToHost, s);
        if ((e = cudaStreamSynchronize(s)) != cudaSuccess) return server_fail(v, e, "hop");
        adm.keep();
        const unsigned long long *off = v->h_out + v->slots;
        /* the new ids, in stages, to their queries */
        for (uint32_t i = 0; i < A; ++i)
            v->state[act[i]].ids.reserve(v->state[act[i]].ids.size() + (off[i + 1] - off[i]));
        uint32_t i = 0;
        for (unsigned long long at = 0; at < off[A]; at += kIdsStage) {
            const unsigned long long end = std::min<unsigned long long>(at + kIdsStage, off[A]);
            cudaMemcpyAsync(v->h_ids, mo.ids + at, sizeof(uint32_t) * (end - at), cudaMemcpyDeviceToHost, s);
            if ((e = cudaStreamSynchronize(s)) != cudaSuccess) return server_fail(v, e, "results");
            for (unsigned long long p = at; p < end;) {
                while (off[i + 1] <= p) ++i;
                const unsigned long long q = std::min(off[i + 1], end);
                std::vector<uint32_t> &ids = v->state[act[i]].ids;
                ids.insert(ids.end(), v->h_ids + (p - at), v->h_ids + (q - at));
                p = q;
            }
        }
        for (uint32_t ai = 0; ai < A; ++ai) {
            SlotState &st = v->state[act[ai]];
            const uint32_t got = (uint32_t)(off[ai + 1] - off[ai]);
            st.hop_end[st.hop] = st.ids.size();
            ++st.hop;
            st.frontier = got;
            st.front_ids = mo.ids + off[ai];
            st.reached += got;
            if (st.hop >= st.hops || got == 0) server_finish(v, st, v->h_out[act[ai]]);
        }
        v->side ^= 1u;
    }
    /* queries admitted with an empty frontier or zero kept blocks finish here */
    for (uint32_t k = 0; k < v->slots; ++k) {
        SlotState &st = v->state[k];
        if (st.busy && st.frontier == 0 && st.hop < st.hops) server_finish(v, st, 0);
    }
    if (n_active) {
        uint32_t n = 0;
        for (const SlotState &st : v->state) n += st.busy ? 1u : 0u;
        *n_active = n;
    }
    if (n_queued) *n_queued = (uint32_t)v->queue.size();
    return GLINT_OK;
}

extern "C" glint_status glint_server_poll(glint_server *v, uint64_t ticket, glint_query_result *r, int *done) {
    if (!v || !done) return GLINT_ERR_INVALID_ARGUMENT;
    auto it = v->done.find(ticket);
    if (it == v->done.end()) {
        *done = 0;
        return GLINT_OK;
    }
    *done = 1;
    if (r) {
        const FinishedQuery &f = it->second;
        r->n = f.ids.size();
        for (uint32_t h = 0; h < kMaxHops; ++h) r->hop_end[h] = f.hop_end[h];
        r->keys_scanned = f.keys_scanned;
        if (r->ids && r->cap) std::memcpy(r->ids, f.ids.data(), sizeof(uint32_t) * std::min<uint64_t>(r->cap, f.ids.size()));
    }
    v->done.erase(it);
    return GLINT_OK;
}

namespace glint {
void server_free_default(glint_ctx *c) {
    if (c->server) glint_server_destroy(c->server);
    c->server = nullptr;
}

void servers_detach(glint_ctx *c) {
    for (glint_server *v : c->servers) {
        server_release(v);
        v->ctx = nullptr;
    }
    c->servers.clear();
}
} // namespace glint

/* a batch through the context's default server: all queries queued, steps
 * until every one has finished */
extern "C" glint_status glint_query_batch(glint_ctx *c, const glint_query *qs, uint32_t nq, glint_query_result *rs) {
    if (!c || (nq && (!qs || !rs))) return GLINT_ERR_INVALID_ARGUMENT;
    for (uint32_t q = 0; q < nq; ++q)
        if ((qs[q].n_seeds && !qs[q].seeds) || qs[q].hops == 0 || qs[q].hops > kMaxHops)
            return GLINT_ERR_INVALID_ARGUMENT;
    cudaSetDevice(c->device);
    cudaError_t e = cudaStreamSynchronize(c->stream);
    if (e != cudaSuccess) {
        c->last_error = std::string("query: ") + cudaGetErrorString(e);
        return GLINT_ERR_CUDA;
    }
    if (!c->server) {
        const glint_status st = glint_server_create(c, 64, &c->server);
        if (st != GLINT_OK) return st;
    }
    glint_server *v = c->server;
    std::vector<uint64_t> tickets(nq);
    for (uint32_t q = 0; q < nq; ++q) glint_server_submit(v, &qs[q], &tickets[q]);
    uint32_t finished = 0;
    std::vector<char> got(nq, 0);
    while (finished < nq) {
        const glint_status st = glint_server_step(v, nullptr, nullptr);
        if (st != GLINT_OK) {
            cancel_queries(tickets, v->queue, v->state, v->done);
            return st;
        }
        for (uint32_t q = 0; q < nq; ++q) {
            if (got[q]) continue;
            int done = 0;
            glint_server_poll(v, tickets[q], &rs[q], &done);
            if (done) {
                got[q] = 1;
                ++finished;
            }
        }
    }
    return GLINT_OK;
}

extern "C" uint32_t glint_store_blocks(const glint_ctx *c) { return c ? (uint32_t)c->ctbs.size() : 0u; }
