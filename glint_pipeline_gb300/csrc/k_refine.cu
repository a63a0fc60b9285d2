/*
 * k_refine.cu -- stages (b) part 2, (c) and (d) part 1 in the plain form:
 * per-leaf candidate enumeration, the reference's FP64 distance test on every
 * candidate, and the meeting-table update.
 *
 * Candidates (tracing/refinement.cpp:19-31): for every check and every stored
 * member of its leaf with pid < member (inside checks) or any member
 * (cross-leaf checks).  p1 is the checking object, whose latitude sets
 * degree_per_meter_longitude in Point::distance (geometry/geometry.h:40-48).
 *
 * Device form: one warp per leaf.  The leaf's stored members (its first
 * min(count, capacity) objects in id order) are staged in shared memory as
 * FP32 offsets from the leaf; the warp runs the inside pairs i < j and then
 * every cross-leaf check that targets the leaf against the staged members
 * (refine_common.cuh).  A pair whose FP32 distance is beyond reach by more
 * than the screen's proven error is ruled out there; every other pair goes
 * through the contact queue and is decided by the FP64 test when the queue is
 * drained, 32 pairs to a warp instruction.  A contact found in the table as it
 * stood at the start of the step is touched there, which is what the
 * reference does for it; a pair not found goes to the new list with its
 * position in the reference's sequential check order as priority.
 *
 * Bound: FP64 issues at 1/64 of the FP32 rate, so the reference's expression
 * on every candidate (two divisions, a square root: about 45 FP64 operations)
 * was the whole kernel.  1M objects, 18.7M candidates, 3.0M contacts, GB300:
 * 4832 us with FP64 on every candidate, 263 us with the bound, the queue and
 * the division-free test (215 us in the form that accepts by the screen too);
 * 100k objects, 1.4M candidates: 525 and 22 us.
 *
 * Duplicate pairs: a cross-leaf pair (a, b) is tested from both sides when a
 * has a check on b's leaf and b one on a's leaf.  The reference's second test
 * only re-touches the entry the first one made; here the test from the larger
 * id is dropped when the other test also passes, so every pair has at most
 * one event per step.
 */
#include <algorithm>
#include <atomic>

#include "refine_common.cuh"

namespace glint {

constexpr int kRefineWarps = 4;

__global__ void __launch_bounds__(32 * kRefineWarps) k_refine_fp64(RefineArgs a) {
    extern __shared__ __align__(64) unsigned char smem_raw[];
    const LeafTile m = leaf_tile(smem_raw + (size_t)(threadIdx.x >> 5) * tile_warp_bytes(a.cap), a.cap);
    RefineTally t;
    uint32_t qn = 0;
    const uint32_t tag = a.cnt->step_tag;
    refine_items<true>(a, m, t, qn, tag);
    refine_flush<true>(a, m.Q, qn, tag, t);
}

/* the warps per block whose leaf tiles and contact queues fit the per-block
 * limit of shared memory (large leaf buffers run with fewer) */
int refine_warps(uint32_t cap) {
    return (int)std::max<size_t>(1, std::min<size_t>(kRefineWarps, kMaxBlockSmem / tile_warp_bytes(cap)));
}
size_t refine_smem_bytes(uint32_t cap) { return (size_t)refine_warps(cap) * tile_warp_bytes(cap); }

RefineArgs refine_args(glint_ctx *c) {
    RefineArgs a;
    a.work = c->d_leaf_work;
    a.grid_start = c->d_grid_start;
    a.grid_count = c->d_grid_count;
    a.sorted = c->d_sorted;
    a.sxy = c->d_sxy;
    a.sm = c->d_sm;
    a.ibox = c->d_ibox;
    a.tstart = c->d_tstart;
    a.tlist = c->d_tlist;
    a.sipos = c->d_sipos;
    a.sfpos = c->d_sfpos;
    a.sc = c->d_sc;
    a.f = c->frame;
    a.info = c->d_info;
    a.rank = c->d_rank;
    a.qstart = c->d_qstart;
    a.qcount = c->d_qcount;
    a.qlist = c->d_qlist;
    a.extra = c->d_rextra;
    a.tab = c->d_tab;
    a.stamp = c->B <= kStampTouchBuckets ? c->d_stamp : nullptr;
    a.newlist = c->d_new;
    a.B = c->B;
    a.Bm = c->Bm;
    a.new_cap = c->new_cap;
    a.cap = c->cap;
    a.chunk = c->chunk;
    a.extra_cap = (uint32_t)std::min<uint64_t>(c->rextra_cap, 0xffffffffu);
    a.ex = make_exact(c);
    a.m_lat = 1.0 / c->dpm_lat;
    a.r2 = c->cfg.reach_distance * c->cfg.reach_distance;
    a.tol = 4.0 * c->cfg.reach_distance * c->band;
    a.cnt = c->d_cnt;
    return a;
}

cudaError_t launch_refine_precision(glint_ctx *c, const RefineArgs &a);

/* the refine stage's pair tests over its work items */
cudaError_t launch_refine_pairs(glint_ctx *c) {
    RefineArgs a = refine_args(c);
    if (c->cfg.precision_mode == 1) return launch_refine_precision(c, a);
    k_refine_fp64<<<152 * 8, 32 * refine_warps(c->cap), refine_smem_bytes(c->cap), c->stream>>>(a);
    return cudaGetLastError();
}

/* The limit is a property of the kernel, shared by every context of the
 * process: it is set to the per-block maximum, and every launch asks for the
 * shared memory its leaf buffer needs. */
void refine_set_attributes(uint32_t cap) {
    (void)cap;
    cudaFuncSetAttribute(k_refine_fp64, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMaxBlockSmem);
}

/* ---- insertion of the step's new pairs -------------------------------------
 * Deterministic linear probing with priority displacement: a pair walking from
 * its home bucket takes an empty bucket, or swaps itself into a bucket held by
 * a pair inserted this step with a larger priority (which then walks on from
 * the next bucket).  Committed pairs are never moved.  The final layout is
 * the one a single thread produces by inserting the pairs one by one in
 * priority order, which is the reference's order (tracing/refinement.cpp:
 * 34-55).  A pair that meets its own committed entry further along (left there
 * when an earlier bucket of its probe run emptied) touches that entry instead,
 * as the reference does when its probe reaches it. */
__device__ inline bool u128_eq(const ulonglong2 &a, const ulonglong2 &b) { return a.x == b.x && a.y == b.y; }

__device__ inline ulonglong2 cas128(TRec *r, ulonglong2 expect, ulonglong2 desired) {
    unsigned __int128 e = ((unsigned __int128)expect.y << 64) | expect.x;
    unsigned __int128 d = ((unsigned __int128)desired.y << 64) | desired.x;
    unsigned __int128 o = atomicCAS(reinterpret_cast<unsigned __int128 *>(r), e, d);
    return make_ulonglong2((unsigned long long)o, (unsigned long long)(o >> 64));
}

__device__ inline void touch_box(TRec &r, const float2 &A, const float2 &Bp) {
    const float ax = A.x, ay = A.y, bx = Bp.x, by = Bp.y;
    uint4 m = *reinterpret_cast<const uint4 *>(r.mbr);
    m.x = min(m.x, min(fenc(ax), fenc(bx)));
    m.y = min(m.y, min(fenc(ay), fenc(by)));
    m.z = max(m.z, max(fenc(ax), fenc(bx)));
    m.w = max(m.w, max(fenc(ay), fenc(by)));
    *reinterpret_cast<uint4 *>(r.mbr) = m;
}

__global__ void __launch_bounds__(256) k_insert(const NewEntry *__restrict__ list, TRec *tab, uint32_t *newline,
                                                uint8_t *stamp,
                                                uint64_t B, uint64_t Bm, uint64_t new_cap,
                                                const float2 *__restrict__ fpos, uint32_t N,
                                                DevCounters *cnt) {
    const unsigned long long n0 = cnt->new_keys;
    const unsigned long long n = n0 < new_cap ? n0 : new_cap;
    const uint8_t st = (uint8_t)cnt->step_tag;
    uint64_t span = 0; /* the farthest placement from a home slot, + 1 */
    for (unsigned long long i = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; i < n;
         i += (unsigned long long)gridDim.x * blockDim.x) {
        ulonglong2 cur = make_ulonglong2(list[i].key | kNewFlag, list[i].prio);
        uint64_t slot = fastmod(cantor(pair_a(cur.x), pair_b(cur.x)), B, Bm), home = slot;
        auto placed = [&]() {
            const uint64_t d = (slot >= home ? slot - home : slot + B - home) + 1;
            span = d > span ? d : span;
        };
        bool done = false;
        /* empty records hold (kEmptyW0, 0), so the first compare-and-swap at a
         * bucket doubles as its read */
        const ulonglong2 empty = make_ulonglong2(kEmptyW0, 0ull);
        for (uint32_t iter = 0; iter < kProbeLimit && !done; ++iter) {
            ulonglong2 seen = empty;
            for (uint32_t retry = 0;; ++retry) {
                if (retry >= kProbeLimit) {
                    atomicOr(&cnt->error_flags, GLINT_EF_TABLE_FULL);
                    done = true;
                    break;
                }
                const unsigned long long plain = cur.x & kPairMask;
                if (seen.x == kEmptyW0) {
                    ulonglong2 prev = cas128(&tab[slot], seen, cur);
                    if (u128_eq(prev, seen)) {
                        placed();
                        atomicOr(&newline[slot >> 7], 1u << ((slot >> 2) & 31));
                        done = true;
                        break;
                    }
                    seen = prev;
                    continue;
                }
                if (seen.x == plain) {
                    /* the carried pair's own committed entry */
                    const uint32_t pa = pair_a(plain), pb = pair_b(plain);
                    if (pa < N && pb < N) touch_box(tab[slot], fpos[pa], fpos[pb]);
                    if (stamp) stamp[slot] = (uint8_t)(kStampTouched + st);
                    else rec_set_tag(tab[slot], st);
                    done = true;
                    break;
                }
                if (seen.x == cur.x) {
                    atomicOr(&cnt->error_flags, GLINT_EF_DUPLICATE_NEW);
                    done = true;
                    break;
                }
                if ((seen.x & kNewFlag) && seen.y > cur.y) {
                    ulonglong2 prev = cas128(&tab[slot], seen, cur);
                    if (u128_eq(prev, seen)) {
                        placed();
                        cur = seen; /* the displaced pair walks on */
                        home = fastmod(cantor(pair_a(cur.x), pair_b(cur.x)), B, Bm);
                        break;
                    }
                    seen = prev;
                    continue;
                }
                break; /* a committed pair or an earlier new pair */
            }
            if (!done) slot = (slot + 1 == B) ? 0 : slot + 1;
        }
        if (!done) atomicOr(&cnt->error_flags, GLINT_EF_TABLE_FULL);
    }
    /* a high-water mark: after the first steps hardly any placement passes it */
    if (span > cnt->probe_span && cnt->probe_span)
        atomicMax(&cnt->probe_span, (unsigned int)(span < 0xffffffffull ? span : 0xffffffffull));
}

cudaError_t launch_insert(glint_ctx *c, uint32_t cur_time) {
    (void)cur_time;
    /* many short blocks: a thread's walk can be long (probe runs,
     * displacements), and with one resident wave of long grid-stride loops
     * the slowest threads set the kernel's end; up to 152 x 128 blocks
     * balance it (5.4 against 7.7 ms at 10M objects), fewer for a small
     * context's new-pair capacity */
    const unsigned blocks = (unsigned)std::min<uint64_t>(152u * 128u, std::max<uint64_t>(152u, c->new_cap / 2048));
    k_insert<<<blocks, 256, 0, c->stream>>>(c->d_new, c->d_tab, c->d_newline,
                                             c->B <= kStampTouchBuckets ? c->d_stamp : nullptr, c->B, c->Bm, c->new_cap, c->d_fpos, c->N,
                                             c->d_cnt);
    return cudaGetLastError();
}

} // namespace glint
