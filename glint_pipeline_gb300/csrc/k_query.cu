/*
 * k_query.cu -- the active contact search (glint_active_search).
 *
 * Reference: with search_multi set, cuda_identify_meetings (cuda/geometry.cu:
 * 605-663) checks every bucket whose meeting is still active (end ==
 * cur_time) and has lasted cur_time - start >= min_meet_time + 1 against the
 * listed ids (search_multi_pid) and appends (pid, target, start, end, mbr)
 * records (search_info_unit, tracing/workbench.h:85-88) with an atomic
 * counter; tracing/process.cpp:465-475 prints them after the step.
 *
 * Device form, run after a step against the table it left, in bucket order,
 * in two ways.
 *
 * By object (k_search_objects, k_search_sort), for lists that are short beside
 * the table: an entry is active exactly when its pair was a contact of the
 * last step, so the contacts of the listed objects are found again from the
 * step's leaf and check lists, one warp per object, and their entries looked up
 * (past slots that emptied since, as far as any entry was ever placed from
 * its home slot); the entries found, at most kFoundMax, are put in bucket order
 * by one block.
 *
 * By bucket (k_search_count, k_search_emit), for the rest: the listed ids
 * become a bitmap of N bits; pass 1 reads the stamp byte of every bucket and
 * the record of occupied buckets, and counts matching sides per 8192-bucket
 * tile; an exclusive scan gives
 * each tile its offset; pass 2 writes the records of tiles that have any.  A
 * warp lists the occupied buckets of its span first, so that its lanes all
 * have a record to read.
 *
 * 256 objects of 2M, 2^27 buckets 6% full: a call took 423 us by bucket, each
 * thread reading the records of 16 consecutive ones, and takes 64 us by object.
 */
#include <algorithm>
#include <cstring>
#include <mutex>

#include "refine_common.cuh"

namespace glint {

constexpr int kSearchThreads = 512;
constexpr int kSearchItems = 16;
constexpr uint32_t kSearchTile = kSearchThreads * kSearchItems;

static uint64_t search_tiles(uint64_t B) { return (B + kSearchTile - 1) / kSearchTile; }

struct SearchArgs {
    const TRec *tab;
    const uint8_t *stamp;
    uint64_t B;
    uint32_t cur_time;
    uint32_t min_plus1;
    const uint32_t *bits;
    uint32_t N;
};

__global__ void __launch_bounds__(256) k_search_set_bits(const uint32_t *__restrict__ pids, uint32_t n,
                                                         uint32_t *__restrict__ bits, uint32_t N) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const uint32_t p = pids[i];
        if (p < N) atomicOr(&bits[p >> 5], 1u << (p & 31));
    }
}

__device__ inline bool listed(const SearchArgs &a, uint32_t p) {
    return p < a.N && ((a.bits[p >> 5] >> (p & 31)) & 1u);
}

/* matching sides of a record (its words w0, w1): bit 0 the lower id, bit 1 the
 * higher id.  Between steps every entry of the table is active: identify took
 * out the ones that the step did not touch. */
__device__ inline uint32_t search_sides(const SearchArgs &a, const ulonglong2 &r) {
    if (r.x == kEmptyW0 || (r.x & kNewFlag)) return 0;
    if (a.cur_time - (uint32_t)r.y < a.min_plus1) return 0;
    return (listed(a, pair_a(r.x)) ? 1u : 0u) | (listed(a, pair_b(r.x)) ? 2u : 0u);
}

constexpr int kSearchWarps = kSearchThreads / 32;
constexpr uint32_t kSearchSpan = kSearchTile / kSearchWarps;
constexpr int kSearchIlp = 4;

/* warp-collective: the occupied buckets of the span from wbase on, in order,
 * into list; returns their number */
__device__ inline uint32_t list_occupied(const SearchArgs &a, uint64_t wbase, uint16_t *list) {
    const int lane = threadIdx.x & 31;
    uint32_t n = 0;
#pragma unroll
    for (uint32_t i = 0; i < kSearchSpan / 512; ++i) {
        /* 16 stamps per lane (the array is padded to whole tiles) */
        const uint32_t off = i * 512 + lane * 16;
        const uint4 v = *reinterpret_cast<const uint4 *>(a.stamp + wbase + off);
        const uint32_t w[4] = {v.x, v.y, v.z, v.w};
        uint32_t bits = 0;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const uint32_t m = __vcmpne4(w[k], 0u) & 0x08040201u;
            bits |= ((m | (m >> 8) | (m >> 16) | (m >> 24)) & 0xfu) << (4 * k);
        }
        uint32_t incl = __popc(bits);
        const uint32_t mine = incl;
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += y;
        }
        uint32_t at = n + incl - mine;
        n += __shfl_sync(0xffffffffu, incl, 31);
        for (; bits; bits &= bits - 1) list[at++] = (uint16_t)(off + __ffs(bits) - 1);
    }
    __syncwarp();
    return n;
}

__global__ void __launch_bounds__(kSearchThreads) k_search_count(SearchArgs a, uint32_t *__restrict__ tile_cnt) {
    __shared__ uint32_t red[kSearchWarps];
    __shared__ uint16_t list[kSearchWarps][kSearchSpan];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const uint64_t wbase = (uint64_t)blockIdx.x * kSearchTile + (uint64_t)wid * kSearchSpan;
    const uint32_t n = list_occupied(a, wbase, list[wid]);
    uint32_t v = 0;
    for (uint32_t r0 = 0; r0 < n; r0 += 32 * kSearchIlp) {
        ulonglong2 rec[kSearchIlp];
#pragma unroll
        for (int u = 0; u < kSearchIlp; ++u) {
            const uint32_t i = r0 + u * 32 + lane;
            rec[u] = make_ulonglong2(kEmptyW0, 0ull);
            if (i < n) rec[u] = *reinterpret_cast<const ulonglong2 *>(&a.tab[wbase + list[wid][i]]);
        }
#pragma unroll
        for (int u = 0; u < kSearchIlp; ++u) v += __popc(search_sides(a, rec[u]));
    }
    v = __reduce_add_sync(0xffffffffu, v);
    if (lane == 0) red[wid] = v;
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t t = 0;
        for (int i = 0; i < kSearchWarps; ++i) t += red[i];
        tile_cnt[blockIdx.x] = t;
    }
}

/* the record of one side of an entry */
__device__ inline glint_search_info search_record(const TRec &r, uint32_t side, uint32_t cur_time) {
    const uint32_t pa = pair_a(r.w0), pb = pair_b(r.w0);
    glint_search_info o;
    o.pid = side ? pb : pa;
    o.target = side ? pa : pb;
    o.start = (uint32_t)r.w1;
    o.end = cur_time;
    for (int k = 0; k < 4; ++k) o.mbr[k] = fdec(r.mbr[k]);
    return o;
}

__global__ void __launch_bounds__(kSearchThreads) k_search_emit(SearchArgs a, const uint32_t *__restrict__ tile_cnt,
                                                                const uint32_t *__restrict__ tile_off,
                                                                glint_search_info *__restrict__ out, uint64_t cap) {
    if (tile_cnt[blockIdx.x] == 0) return; /* uniform per block */
    __shared__ uint32_t ws[kSearchWarps];
    __shared__ uint16_t list[kSearchWarps][kSearchSpan];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const uint64_t wbase = (uint64_t)blockIdx.x * kSearchTile + (uint64_t)wid * kSearchSpan;
    const uint32_t n = list_occupied(a, wbase, list[wid]);
    uint64_t pos = 0;
    for (int pass = 0; pass < 2; ++pass) {
        uint32_t v = 0;
        for (uint32_t r0 = 0; r0 < n; r0 += 32) {
            const uint32_t i = r0 + lane;
            ulonglong2 rec = make_ulonglong2(kEmptyW0, 0ull);
            if (i < n) rec = *reinterpret_cast<const ulonglong2 *>(&a.tab[wbase + list[wid][i]]);
            const uint32_t m = search_sides(a, rec);
            if (pass == 0) {
                v += __popc(m);
                continue;
            }
            uint32_t incl = __popc(m);
            const uint32_t mine = incl;
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += y;
            }
            uint64_t at = pos + incl - mine;
            pos += __shfl_sync(0xffffffffu, incl, 31);
            if (!m) continue;
            const TRec r = a.tab[wbase + list[wid][i]];
            for (uint32_t side = 0; side < 2; ++side) {
                if (!(m & (1u << side))) continue;
                if (at < cap) out[at] = search_record(r, side, a.cur_time);
                ++at;
            }
        }
        if (pass == 1) break;
        v = __reduce_add_sync(0xffffffffu, v);
        if (lane == 0) ws[wid] = v;
        __syncthreads();
        pos = tile_off[blockIdx.x];
        for (int w = 0; w < wid; ++w) pos += ws[w];
    }
}

/* ---- by object ------------------------------------------------------------ */
constexpr uint32_t kFoundMax = 4096;

struct ObjectSearch {
    RefineArgs r;              /* the step's lists and the table (leaf counts from the segment starts: the
                                  schema update clears those of grids it frees) */
    SearchArgs s;
    unsigned long long *found; /* [kFoundMax] bucket * 2 + side */
    unsigned int *n_found;
};

/* p1 the checking object, p2 the member, as leaf-major ranks */
__device__ inline bool within_reach(const RefineArgs &a, uint32_t r1, uint32_t r2) {
    const longlong2 A = a.sipos[r1], B = a.sipos[r2];
    const Screen sc = make_screen(__fmaf_rn(0.0f, a.sc[r2], a.sc[r1]), a.f);
    const int in = fx_screen(A.x - B.x, A.y - B.y, sc, a.f.cy);
    return in < 0 ? pair_exact(a.sxy, r1, r2, a.ex) : in != 0;
}

/* the listed object p meets m: its entry, if it has lasted long enough */
__device__ inline void found_contact(const ObjectSearch &o, uint32_t p, uint32_t m) {
    const unsigned long long pw = pw_of(p, m);
    uint64_t slot = home_slot(o.r, pw);
    const uint32_t span = o.r.cnt->probe_span;
    for (uint32_t d = 0; d < span; ++d) {
        const ulonglong2 k = *reinterpret_cast<const ulonglong2 *>(&o.r.tab[slot]);
        if (k.x == pw) {
            if (o.s.cur_time - (uint32_t)k.y < o.s.min_plus1) return;
            const uint32_t i = atomicAdd(o.n_found, 1u);
            if (i < kFoundMax) o.found[i] = slot * 2 + (pair_a(pw) == p ? 0u : 1u);
            return;
        }
        slot = slot + 1 == o.r.B ? 0 : slot + 1;
    }
}

/* one warp per listed object: its own leaf's members, the members of the
 * leaves it checks, and the objects that check its leaf (a contact found from
 * both sides, or an object listed twice, is found twice) */
__global__ void __launch_bounds__(128) k_search_objects(ObjectSearch o, const uint32_t *__restrict__ pids,
                                                        uint32_t npids) {
    const RefineArgs &a = o.r;
    const int lane = threadIdx.x & 31;
    for (uint32_t i = (blockIdx.x * blockDim.x + threadIdx.x) / 32; i < npids; i += gridDim.x * blockDim.x / 32) {
        const uint32_t p = pids[i];
        if (p >= o.s.N) continue;
        const uint32_t rank = a.rank[p].x, r = rank & ~kDropped, g = a.info[r].y;
        const uint32_t s0 = a.grid_start[g], k = min(a.grid_start[g + 1] - s0, a.cap);
        const bool stored = !(rank & kDropped);
        for (uint32_t j = lane; stored && j < k; j += 32) {
            const uint32_t m = s0 + j;
            if (m != r && within_reach(a, min(r, m), max(r, m))) found_contact(o, p, a.sorted[m]);
        }
        const uint32_t nq = a.qcount[p], q0 = a.qstart[p];
        for (uint32_t q = 0; q < nq; ++q) {
            const uint32_t h = a.qlist[q0 + q];
            const uint32_t h0 = a.grid_start[h], hk = min(a.grid_start[h + 1] - h0, a.cap);
            for (uint32_t j = lane; j < hk; j += 32)
                if (within_reach(a, r, h0 + j)) found_contact(o, p, a.sorted[h0 + j]);
        }
        const uint32_t tb = a.tstart[g], te = a.tstart[g + 1];
        for (uint32_t t = tb + lane; stored && t < te; t += 32) {
            const uint32_t q = a.tlist[t].x;
            if (within_reach(a, a.rank[q].x & ~kDropped, r)) found_contact(o, p, q);
        }
    }
}

/* one block: the entries found, in bucket order and each once; n = their
 * number, or all ones when there were more than kFoundMax */
__global__ void __launch_bounds__(1024) k_search_sort(ObjectSearch o, glint_search_info *__restrict__ out,
                                                      uint64_t cap, unsigned long long *n) {
    __shared__ unsigned long long key[kFoundMax];
    __shared__ uint32_t ws[32];
    const uint32_t found = *o.n_found;
    if (found > kFoundMax) {
        if (threadIdx.x == 0) *n = ~0ull;
        return;
    }
    uint32_t P = 32;
    while (P < found) P <<= 1;
    for (uint32_t i = threadIdx.x; i < P; i += blockDim.x) key[i] = i < found ? o.found[i] : ~0ull;
    __syncthreads();
    for (uint32_t k = 2; k <= P; k <<= 1)
        for (uint32_t j = k >> 1; j > 0; j >>= 1) {
            for (uint32_t i = threadIdx.x; i < P; i += blockDim.x) {
                const uint32_t l = i ^ j;
                if (l > i) {
                    const unsigned long long x = key[i], y = key[l];
                    if ((x > y) == ((i & k) == 0)) {
                        key[i] = y;
                        key[l] = x;
                    }
                }
            }
            __syncthreads();
        }
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    uint32_t before = 0;
    for (uint32_t base = 0; base < found; base += blockDim.x) {
        const uint32_t i = base + threadIdx.x;
        const bool mine = i < found && (i == 0 || key[i] != key[i - 1]);
        const unsigned m = __ballot_sync(0xffffffffu, mine);
        if (lane == 0) ws[wid] = __popc(m);
        __syncthreads();
        uint32_t at = before, all = 0;
        for (int w = 0; w < 32; ++w) {
            if (w < wid) at += ws[w];
            all += ws[w];
        }
        at += __popc(m & ((1u << lane) - 1u));
        if (mine && at < cap) out[at] = search_record(o.r.tab[key[i] >> 1], (uint32_t)(key[i] & 1), o.s.cur_time);
        before += all;
        __syncthreads();
    }
    if (threadIdx.x == 0) *n = before;
}

__global__ void k_search_total(const uint32_t *__restrict__ tile_off, uint64_t tiles, unsigned long long *n) {
    *n = tile_off[tiles];
}

SearchArgs search_args(const glint_ctx *c, const uint32_t *bits) {
    SearchArgs a;
    a.tab = c->d_tab;
    a.stamp = c->d_stamp;
    a.B = c->B;
    a.cur_time = c->last_time;
    a.min_plus1 = c->cfg.min_meet_time + 1;
    a.bits = bits;
    a.N = c->N;
    return a;
}

/* the search on the context's stream with caller-provided scratch:
 * bits[(N + 31) / 32] (cleared here), tile_cnt / tile_off [tiles + 1] and a
 * scan that maps tile_cnt -> tile_off */
template <class Scan>
cudaError_t launch_active_search(const glint_ctx *c, uint32_t *bits, uint32_t *tile_cnt, uint32_t *tile_off,
                                 Scan scan, const uint32_t *d_pids, uint32_t npids, glint_search_info *d_out,
                                 uint64_t cap, unsigned long long *d_n) {
    cudaStream_t s = c->stream;
    const uint64_t tiles = search_tiles(c->B);
    cudaError_t e = cudaMemsetAsync(bits, 0, sizeof(uint32_t) * (((size_t)c->N + 31) / 32), s);
    if (e != cudaSuccess) return e;
    if (npids) k_search_set_bits<<<grid_for(npids, 256, 152u * 4u), 256, 0, s>>>(d_pids, npids, bits, c->N);
    const SearchArgs a = search_args(c, bits);
    k_search_count<<<(unsigned)tiles, kSearchThreads, 0, s>>>(a, tile_cnt);
    if ((e = scan(tile_cnt, tile_off, tiles, s)) != cudaSuccess) return e;
    if (cap) k_search_emit<<<(unsigned)tiles, kSearchThreads, 0, s>>>(a, tile_cnt, tile_off, d_out, cap);
    k_search_total<<<1, 1, 0, s>>>(tile_off, tiles, d_n);
    return cudaGetLastError();
}

} // namespace glint

using namespace glint;

namespace {

template <class T>
cudaError_t grow(T **p, uint64_t &have, uint64_t need) {
    if (need <= have && *p) return cudaSuccess;
    if (*p) cudaFree(*p);
    *p = nullptr;
    have = 0;
    cudaError_t e = cudaMalloc((void **)p, sizeof(T) * (need ? need : 1));
    if (e == cudaSuccess) have = need;
    return e;
}

/* Which way: an object costs its contacts and their entries, a bucket its
 * stamp and, where occupied, its record.  The two meet at about B / 2000
 * objects (2^23 buckets, 200k objects: 4000 by object 76 us a call, 8000 by
 * bucket 71 us), and beyond 2048 objects the entries tend to be more than one
 * block orders (2^27 buckets, 2M objects: 2000 by object 102 us; 4000, found to
 * be too many and then read by bucket, 339 us).  Entries far from their home
 * slots (a table near its capacity) make each look long: past 1024 slots the
 * buckets are read. */
bool search_by_object(const glint_ctx *c, uint32_t npids) {
    const uint32_t span = c->h_cnt->probe_span;
    return c->step_lists && npids && npids <= 2048 && (uint64_t)npids * 2000 < c->B && span && span <= 1024;
}

cudaError_t launch_object_search(glint_ctx *c, uint32_t npids, uint64_t cap) {
    cudaStream_t s = c->stream;
    cudaError_t e = cudaSuccess;
    if (!c->d_qfound) e = cudaMalloc((void **)&c->d_qfound, sizeof(unsigned long long) * (kFoundMax + 1));
    if (e != cudaSuccess) return e;
    ObjectSearch o;
    o.r = refine_args(c);
    o.r.ex.ambiguous = nullptr; /* the step's counters stay the step's */
    o.r.ex.rechecks = nullptr;
    o.s = search_args(c, nullptr);
    o.found = c->d_qfound;
    o.n_found = reinterpret_cast<unsigned int *>(c->d_qfound + kFoundMax);
    if ((e = cudaMemsetAsync(o.n_found, 0, sizeof(unsigned int), s)) != cudaSuccess) return e;
    k_search_objects<<<grid_for(npids, 4, 152u * 16u), 128, 0, s>>>(o, c->d_qpids, npids);
    k_search_sort<<<1, 1024, 0, s>>>(o, c->d_qout, cap, c->d_qn);
    return cudaGetLastError();
}

} // namespace

extern "C" glint_status glint_active_search(glint_ctx *c, const uint32_t *pids, uint32_t npids, glint_search_info *out,
                                            uint64_t cap, uint64_t *n) {
    if (!c || (npids && !pids) || (cap && !out)) return GLINT_ERR_INVALID_ARGUMENT;
    if (serve_only_refused(c, "active search")) return GLINT_ERR_STATE;
    if (c->step_index == 0) {
        c->last_error = "active search before the first step";
        return GLINT_ERR_STATE;
    }
    cudaSetDevice(c->device);
    cudaError_t e = cudaStreamSynchronize(c->stream);
    const uint64_t words = ((uint64_t)c->N + 31) / 32;
    if (e == cudaSuccess) e = grow(&c->d_qpids, c->qpids_cap, std::max<uint64_t>(npids, 1));
    if (e == cudaSuccess) e = grow(&c->d_qout, c->qout_cap, std::max<uint64_t>(cap, 1));
    if (e == cudaSuccess && !c->d_qn) e = cudaMalloc((void **)&c->d_qn, sizeof(unsigned long long));
    if (e == cudaSuccess && npids)
        e = cudaMemcpyAsync(c->d_qpids, pids, sizeof(uint32_t) * npids, cudaMemcpyHostToDevice, c->stream);
    unsigned long long found = ~0ull;
    auto fetch = [&]() {
        if (e == cudaSuccess)
            e = cudaMemcpyAsync(&found, c->d_qn, sizeof(found), cudaMemcpyDeviceToHost, c->stream);
        if (e == cudaSuccess) e = cudaStreamSynchronize(c->stream);
    };
    if (e == cudaSuccess && search_by_object(c, npids)) {
        e = launch_object_search(c, npids, cap);
        fetch();
    }
    /* by bucket, also when more entries were found than one block orders */
    if (e == cudaSuccess && found == ~0ull) e = grow(&c->d_qbits, c->qbits_cap, words);
    if (e == cudaSuccess && found == ~0ull) {
        void *tmp = c->d_scan_tmp;
        auto scan = [tmp](const uint32_t *in, uint32_t *o, uint64_t m, cudaStream_t s) {
            return scan_u32(in, o, m, tmp, s);
        };
        e = launch_active_search(c, c->d_qbits, c->d_tile_cnt, c->d_tile_off, scan, c->d_qpids, npids, c->d_qout, cap,
                                 c->d_qn);
        fetch();
    }
    if (e == cudaSuccess && found && cap)
        e = cudaMemcpy(out, c->d_qout, sizeof(glint_search_info) * std::min<uint64_t>(found, cap),
                       cudaMemcpyDeviceToHost);
    if (e != cudaSuccess) {
        c->last_error = std::string("active search: ") + cudaGetErrorString(e);
        return e == cudaErrorMemoryAllocation ? GLINT_ERR_OUT_OF_MEMORY : GLINT_ERR_CUDA;
    }
    if (n) *n = found;
    return GLINT_OK;
}

/* ---- allocation-free variant --------------------------------------------
 * glint_active_search_noalloc takes device arrays and keeps its scratch in
 * one fixed-size device array of this library: the id bitmap (objects up to
 * kNaMaxObjects) and the per-tile counts and offsets (buckets up to
 * kNaMaxTiles * 8192).  Its address is looked up once per device while a
 * context is created on it; the call itself allocates nothing. */
namespace glint {

constexpr uint32_t kNaMaxObjects = 1u << 24;                 /* 16.7M objects: 2 MB of bits */
constexpr uint32_t kNaMaxTiles = 1u << 17;                   /* 2^30 buckets: 2 x 512 KB */
constexpr size_t kNaBitsWords = kNaMaxObjects / 32;
constexpr size_t kNaTileWords = (size_t)kNaMaxTiles + 64;    /* tiles + 1, padded to 256 B */
constexpr size_t kNaWords = kNaBitsWords + 2 * kNaTileWords;
constexpr int kNaMaxDevices = 64;

static __device__ __align__(256) uint32_t g_noalloc_scratch[kNaWords];

std::mutex g_na_mutex;
uint32_t *g_na_ptr[kNaMaxDevices];
cudaError_t g_na_status[kNaMaxDevices];
bool g_na_done[kNaMaxDevices];

/* exclusive scan of n (<= kNaMaxTiles) values by one block, no scratch;
 * out[n] receives the total, so out has n + 1 words and in only n are read */
__global__ void __launch_bounds__(1024) k_scan_one_block(const uint32_t *__restrict__ in, uint32_t *__restrict__ out,
                                                         uint64_t n) {
    __shared__ uint32_t ws[32];
    __shared__ uint32_t carry;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    if (threadIdx.x == 0) carry = 0;
    __syncthreads();
    for (uint64_t base = 0; base < n; base += blockDim.x) {
        const uint64_t i = base + threadIdx.x;
        const uint32_t v = i < n ? in[i] : 0u;
        uint32_t x = v;
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31) ws[wid] = x;
        __syncthreads();
        if (wid == 0) {
            uint32_t s = ws[lane];
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, s, o);
                if (lane >= o) s += y;
            }
            ws[lane] = s;
        }
        __syncthreads();
        const uint32_t excl = carry + (wid ? ws[wid - 1] : 0u) + x - v;
        if (i < n) out[i] = excl;
        __syncthreads();
        if (threadIdx.x == 0) carry += ws[31];
        __syncthreads();
    }
    if (threadIdx.x == 0) out[n] = carry;
}

/* looks up the scratch address on the current device; run by every
 * glint_create, so a context created after a device reset sees the array's
 * address in the device's new CUDA context */
cudaError_t noalloc_setup(int device) {
    if (device < 0 || device >= kNaMaxDevices) return cudaErrorInvalidDevice;
    std::lock_guard<std::mutex> lock(g_na_mutex);
    void *p = nullptr;
    g_na_status[device] = cudaGetSymbolAddress(&p, g_noalloc_scratch);
    g_na_ptr[device] = g_na_status[device] == cudaSuccess ? static_cast<uint32_t *>(p) : nullptr;
    g_na_done[device] = true;
    return g_na_status[device];
}

} // namespace glint

extern "C" glint_status glint_active_search_noalloc(glint_ctx *c, const uint32_t *d_pids, uint32_t npids,
                                                    glint_search_info *d_out, uint64_t cap, uint64_t *d_n) {
    if (!c || (npids && !d_pids) || (cap && !d_out) || !d_n) return GLINT_ERR_INVALID_ARGUMENT;
    if (serve_only_refused(c, "active search")) return GLINT_ERR_STATE;
    if (c->step_index == 0) {
        c->last_error = "active search before the first step";
        return GLINT_ERR_STATE;
    }
    if (c->N > kNaMaxObjects || search_tiles(c->B) > kNaMaxTiles) {
        c->last_error = "glint_active_search_noalloc: context larger than its fixed scratch (objects <= 2^24, "
                        "buckets <= 2^30); use glint_active_search";
        return GLINT_ERR_UNSUPPORTED;
    }
    uint32_t *base = nullptr;
    cudaError_t st = cudaErrorInvalidDevice;
    {
        std::lock_guard<std::mutex> lock(g_na_mutex);
        if (c->device >= 0 && c->device < kNaMaxDevices && g_na_done[c->device]) {
            st = g_na_status[c->device];
            base = g_na_ptr[c->device];
        }
    }
    if (st != cudaSuccess || !base) {
        c->last_error = std::string("glint_active_search_noalloc: scratch lookup failed: ") + cudaGetErrorString(st);
        return GLINT_ERR_CUDA;
    }
    cudaSetDevice(c->device);
    uint32_t *bits = base;
    uint32_t *tile_cnt = base + kNaBitsWords;
    uint32_t *tile_off = tile_cnt + kNaTileWords;
    auto scan = [](const uint32_t *in, uint32_t *o, uint64_t m, cudaStream_t s) {
        k_scan_one_block<<<1, 1024, 0, s>>>(in, o, m);
        return cudaGetLastError();
    };
    static_assert(sizeof(uint64_t) == sizeof(unsigned long long), "u64");
    const cudaError_t e = launch_active_search(c, bits, tile_cnt, tile_off, scan, d_pids, npids, d_out, cap,
                                               reinterpret_cast<unsigned long long *>(d_n));
    if (e != cudaSuccess) {
        c->last_error = std::string("glint_active_search_noalloc: ") + cudaGetErrorString(e);
        return GLINT_ERR_CUDA;
    }
    return GLINT_OK;
}

