/*
 * refine_common.cuh -- the pair tests and the contact queue shared by the
 * refine kernels: a warp stages a leaf's members in shared memory, screens
 * pairs on FP32 offsets from the leaf, compacts what the screen leaves over
 * with a warp ballot into a per-warp shared queue, and applies the queue to
 * the meeting table 64 at a time.
 */
#ifndef GLINT_REFINE_COMMON_CUH_
#define GLINT_REFINE_COMMON_CUH_

#include "glint_internal.cuh"

namespace glint {

constexpr int kQueue = 96;      /* a drain of 64 plus one enqueue of up to 32 */
constexpr uint32_t kDrainAt = 64;
constexpr uint32_t kProbeLimit = 1u << 22;

struct __align__(16) QEntry {
    unsigned long long pw;     /* pair word (a << 32) | b, a < b */
    unsigned long long prio;   /* position in the reference's check order */
    /* screened form: the two points, rounded to f32; FP64 form: the
     * leaf-major ranks of the checking object and of the member, and whether
     * the member may check the pair too */
    uint4 v;
};

struct RefineArgs {
    const uint32_t *work;
    const uint32_t *grid_start;
    const uint32_t *grid_count;
    const uint32_t *sorted;
    const double2 *sxy;
    const double *sm;          /* FP64 form: metres per degree of longitude, leaf-major */
    const uint32_t *tstart;
    const uint2 *tlist;
    const longlong2 *sipos;    /* fixed-point coordinates, leaf-major */
    const float2 *sfpos;       /* FP32 coordinates, leaf-major */
    const float *sc;           /* screening scale cx, leaf-major */
    const uint2 *info;         /* by rank: .., leaf grid */
    const uint2 *rank;         /* by object id: leaf-major rank (kDropped: not stored), leaf node */
    const uint32_t *qstart, *qcount;
    const uint32_t *qlist;
    const IBox *ibox;
    const uint2 *extra;        /* (leaf, chunk) items beyond each leaf's first chunk */
    TRec *tab;
    uint8_t *stamp;            /* null: a touch is a tag in the record */
    NewEntry *newlist;
    uint64_t B, Bm, new_cap;
    uint32_t cap;
    uint32_t chunk;            /* cross-leaf checks per work item */
    uint32_t extra_cap;        /* entries of `extra` */
    Frame f;
    double m_lat;              /* metres per degree of latitude */
    double r2;                 /* r^2 */
    double tol;                /* half-width of the FP64 test's band around r^2 */
    ExactCtx ex;
    DevCounters *cnt;
};

/* The table as it stood at the start of the step: keys do not change while
 * the refine kernels run.  Found -> touch the entry (tag, f32 box; each pair
 * has at most one event per step, so the box needs no atomics).  Not found
 * before an empty slot -> the pair is new this step.  The walk starts at the
 * home slot, whose key word and box the caller has already loaded. */
__device__ inline bool table_touch_from(const RefineArgs &a, const QEntry &q, uint64_t slot, unsigned long long w0,
                                        uint4 m, uint32_t tag) {
    for (uint32_t probe = 0; probe < kProbeLimit; ++probe) {
        if (w0 == q.pw) {
            const uint32_t x1 = fenc(__uint_as_float(q.v.x)), y1 = fenc(__uint_as_float(q.v.y));
            const uint32_t x2 = fenc(__uint_as_float(q.v.z)), y2 = fenc(__uint_as_float(q.v.w));
            const uint32_t lx = min(x1, x2), hx = max(x1, x2);
            const uint32_t ly = min(y1, y2), hy = max(y1, y2);
            if (lx < m.x || ly < m.y || hx > m.z || hy > m.w) {
                m.x = min(m.x, lx);
                m.y = min(m.y, ly);
                m.z = max(m.z, hx);
                m.w = max(m.w, hy);
                *reinterpret_cast<uint4 *>(a.tab[slot].mbr) = m;
            }
            if (a.stamp) a.stamp[slot] = (uint8_t)(kStampTouched + tag);
            else rec_set_tag(a.tab[slot], tag);
            return false;
        }
        if (w0 == kEmptyW0) return true;
        slot = (slot + 1 == a.B) ? 0 : slot + 1;
        w0 = a.tab[slot].w0;
        m = *reinterpret_cast<const uint4 *>(a.tab[slot].mbr);
    }
    atomicOr(&a.cnt->error_flags, GLINT_EF_TABLE_FULL);
    return false;
}

__device__ inline uint64_t home_slot(const RefineArgs &a, unsigned long long pw) {
    return fastmod(cantor(pair_a(pw), pair_b(pw)), a.B, a.Bm);
}

/* warp-collective: the lanes whose pair is new append it to the new list */
__device__ inline void append_new(const RefineArgs &a, bool isnew, const QEntry &q) {
    const int lane = threadIdx.x & 31;
    const unsigned m = __ballot_sync(0xffffffffu, isnew);
    if (!m) return;
    unsigned long long off = 0;
    const int leader = __ffs(m) - 1;
    if (lane == leader) off = atomicAdd(&a.cnt->new_keys, (unsigned long long)__popc(m));
    off = __shfl_sync(0xffffffffu, off, leader);
    if (isnew) {
        const unsigned long long idx = off + __popc(m & ((1u << lane) - 1u));
        if (idx < a.new_cap) {
            a.newlist[idx].key = q.pw;
            a.newlist[idx].prio = q.prio;
        } else {
            atomicOr(&a.cnt->error_flags, GLINT_EF_NEW_OVERFLOW);
        }
    }
}

/* a warp's tests and contacts of one context, added to its totals on flush */
struct RefineTally {
    unsigned long long cand = 0, hits = 0;
    uint32_t band = 0;
};

/* the reference's FP64 test of two leaf-major ranks, p1 the checking object;
 * out of line, so that none of its FP64 work is scheduled on the common path */
static __device__ __noinline__ bool pair_exact(const double2 *__restrict__ sxy, uint32_t r1, uint32_t r2,
                                        const ExactCtx &ex) {
    const double2 P = sxy[r1], M = sxy[r2];
    return point_le_exact(P.x, P.y, M.x, M.y, dpm_lon_fast(P.y), ex);
}

/* does object obj have a cross-leaf check on grid gid */
__device__ inline bool has_check(const RefineArgs &a, uint32_t obj, uint32_t gid) {
    const uint32_t n = a.qcount[obj];
    if (!n) return false;
    const uint32_t b = a.qstart[obj], e = b + n;
    for (uint32_t k = b; k < e; ++k)
        if (a.qlist[k] == gid) return true;
    return false;
}

/* The FP64 form's test: the squared distance in metres, in FP64 without the
 * reference's two divisions and square root (about 8 FP64 operations instead
 * of 45; FP64 issues at 1/64 of the FP32 rate).  Its error is at most
 * 2^-41 of the result (the longitude scale's 2^-43 twice, metres_per_degree,
 * and a few 2^-52), the band around r^2 is 2^-36 of it, so outside the band
 * its decision is the reference's; inside, the reference's own expression
 * decides.  The band contains every pair that point_le_exact re-takes with
 * the correctly rounded sin (|d - r| <= 2^-38 r), so that count stays. */
__device__ inline bool pair_fp64(const RefineArgs &a, uint32_t r1, uint32_t r2) {
    const double2 P = a.sxy[r1], M = a.sxy[r2];
    const double dx = __dmul_rn(__dsub_rn(P.x, M.x), a.sm[r1]), dy = __dmul_rn(__dsub_rn(P.y, M.y), a.m_lat);
    const double d = __dsub_rn(__fma_rn(dx, dx, __dmul_rn(dy, dy)), a.r2);
    /* |d| against the band as integers (FP64 compares use the same narrow
     * pipe); a NaN is no contact in the reference */
    const unsigned long long b = (unsigned long long)__double_as_longlong(d), m = b & 0x7fffffffffffffffull;
    if (m > (unsigned long long)__double_as_longlong(a.tol)) return (b >> 63) && m <= 0x7ff0000000000000ull;
    return pair_exact(a.sxy, r1, r2, a.ex);
}

/* FP64 form: is this queued pair a contact, and this its only event?  Fills
 * in the two points. */
__device__ inline bool queued_contact(const RefineArgs &a, QEntry &q, RefineTally &t) {
    const uint32_t r1 = q.v.x, r2 = q.v.y;
    if (!pair_fp64(a, r1, r2)) return false;
    ++t.hits;
    if (q.v.z) {
        /* the member's own check of this pair comes first in the reference's
         * order; keep only one event */
        const uint32_t qid = (uint32_t)(q.prio >> 36) & 0x7ffffffu;
        const uint32_t mid = pair_a(q.pw) == qid ? pair_b(q.pw) : pair_a(q.pw);
        if (has_check(a, mid, a.info[r1].y) && pair_fp64(a, r2, r1)) return false;
    }
    const float2 A = a.sfpos[r1], B = a.sfpos[r2];
    q.v = make_uint4(__float_as_uint(A.x), __float_as_uint(A.y), __float_as_uint(B.x), __float_as_uint(B.y));
    return true;
}

/* warp-collective: process queue entries [0, n), two per lane, with both
 * home records requested before either is used (the table is far larger
 * than L2, so each is a DRAM round trip) */
template <bool kFp64>
__device__ inline void drain_queue(const RefineArgs &a, QEntry *Q, uint32_t n, uint32_t tag, RefineTally &t) {
    const int lane = threadIdx.x & 31;
    for (uint32_t base = 0; base < n; base += 64) {
        const uint32_t e0 = base + lane, e1 = base + 32 + lane;
        bool v0 = e0 < n, v1 = e1 < n;
        QEntry q0, q1;
        uint64_t s0 = 0, s1 = 0;
        if (v0) {
            q0 = Q[e0];
            if (kFp64) v0 = queued_contact(a, q0, t);
        }
        if (v1) {
            q1 = Q[e1];
            if (kFp64) v1 = queued_contact(a, q1, t);
        }
        if (v0) s0 = home_slot(a, q0.pw);
        if (v1) s1 = home_slot(a, q1.pw);
        unsigned long long w00 = 0, w01 = 0;
        uint4 m0 = make_uint4(0, 0, 0, 0), m1 = m0;
        if (v0) {
            w00 = a.tab[s0].w0;
            m0 = *reinterpret_cast<const uint4 *>(a.tab[s0].mbr);
        }
        if (v1) {
            w01 = a.tab[s1].w0;
            m1 = *reinterpret_cast<const uint4 *>(a.tab[s1].mbr);
        }
        const bool n0 = v0 && table_touch_from(a, q0, s0, w00, m0, tag);
        const bool n1 = v1 && table_touch_from(a, q1, s1, w01, m1, tag);
        append_new(a, n0, q0);
        append_new(a, n1, q1);
    }
    __syncwarp();
}

/* warp-collective, after some lane has queued an entry: drains a full queue */
template <bool kFp64>
__device__ inline void drain_if_full(const RefineArgs &a, QEntry *Q, uint32_t &qn, uint32_t added, uint32_t tag,
                                     RefineTally &t) {
    const int lane = threadIdx.x & 31;
    qn += added;
    __syncwarp();
    if (qn >= kDrainAt) {
        drain_queue<kFp64>(a, Q, kDrainAt, tag, t);
        const uint32_t rest = qn - kDrainAt;
        if ((uint32_t)lane < rest) Q[lane] = Q[kDrainAt + lane];
        __syncwarp();
        qn = rest;
    }
}

/* Work items: a leaf's inside pairs with its first `chunk` cross-leaf
 * checks, and one item per further chunk of its checks.  Dense leaves are
 * the target of thousands of checks; split into chunks they spread over the
 * warps instead of leaving a long tail on one.  Every event carries its
 * position in the reference's order, so the split does not change results. */
/* warp-collective: the next item, extra chunks first (the long work first);
 * false when none is left */
__device__ inline bool claim_item(const RefineArgs &a, uint32_t nwork, uint32_t n_extra, bool &extra_done,
                                  uint32_t &g, uint32_t &chunk) {
    const int lane = threadIdx.x & 31;
    uint32_t v = 0, kind = 0;
    if (lane == 0) {
        if (!extra_done) {
            v = atomicAdd(&a.cnt->extra_next, 1u);
            if (v < n_extra && v < a.extra_cap) kind = 1;
        }
        if (kind == 0) {
            v = atomicAdd(&a.cnt->work_next, 1u);
            kind = v < nwork ? 2u : 0u;
        }
    }
    kind = __shfl_sync(0xffffffffu, kind, 0);
    v = __shfl_sync(0xffffffffu, v, 0);
    if (kind == 1) {
        const uint2 e = a.extra[v];
        g = e.x;
        chunk = e.y;
        return true;
    }
    extra_done = true;
    if (kind == 2) {
        g = a.work[v];
        chunk = 0;
        return true;
    }
    return false;
}

/* the cross-leaf checks of one item */
__device__ inline void item_checks(const RefineArgs &a, uint32_t g, uint32_t chunk, uint32_t &tb, uint32_t &te) {
    const uint32_t b = a.tstart[g], e = a.tstart[g + 1];
    tb = b + chunk * a.chunk;
    te = tb + a.chunk < e ? tb + a.chunk : e;
    if (tb > e) tb = e;
}

__device__ inline unsigned long long pw_of(uint32_t p, uint32_t q) { return p < q ? pair_word(p, q) : pair_word(q, p); }

/* ---- pair screening on leaf-relative offsets -------------------------------
 * A staged member's offset from the leaf's first member is held in FP32, in
 * fixed-point units: a = fl(X - X0), |a - (X - X0)| <= u M with u = 2^-24 and
 * M the largest such offset.  The difference of two offsets is then within
 * 2 u M + u |d| of the exact integer difference; the second term is the one
 * conversion rounding that the band of glint_device.cuh already has, and the
 * first adds at most 2 r (2 u)(Mx cx + My cy) to q near the threshold.  The
 * band is widened by twice that: 8 r u (Mx cx + My cy).  (A second-order term
 * is smaller by u M c / r: 0.2% at a leaf 60 km wide.)  So the screen costs
 * two FP32 subtractions per pair where 64-bit differences and their
 * conversions cost about thirty instructions.  A NaN (an offset or a scale
 * out of range) compares false and leaves the pair to the exact test. */
struct LeafTile {
    float2 *pos;               /* offsets */
    float2 *cb;                /* metres per unit along x, guard band */
    float2 *xy;                /* f32 coordinates (screened form) */
    uint32_t *id;
    QEntry *Q;
};

__host__ __device__ inline size_t tile_warp_bytes(uint32_t cap) {
    const size_t per_warp = sizeof(QEntry) * kQueue + (size_t)cap * 28;
    return (per_warp + 63) & ~(size_t)63;
}

__device__ inline LeafTile leaf_tile(unsigned char *base, uint32_t cap) {
    LeafTile m;
    m.Q = reinterpret_cast<QEntry *>(base);
    m.pos = reinterpret_cast<float2 *>(m.Q + kQueue);
    m.cb = m.pos + cap;
    m.xy = m.cb + cap;
    m.id = reinterpret_cast<uint32_t *>(m.xy + cap);
    return m;
}

/* the staged leaf: its origin and the largest offsets of its members */
struct LeafOrigin {
    uint32_t g = ~0u;
    long long X0 = 0, Y0 = 0;
    float Mx = 0.f, My = 0.f;
};

__device__ inline float pair_band(const Frame &f, float c, float mx, float my) {
    return f.band0 + f.band1 * (c + f.cy) + (f.band1 * 1.1920929e-7f) * (mx * c + my * f.cy);
}

/* warp-collective: stage the k stored members of leaf g */
__device__ inline void stage_leaf(const RefineArgs &a, uint32_t g, uint32_t s0, uint32_t k, const LeafTile &m,
                                  LeafOrigin &o, bool with_xy) {
    const int lane = threadIdx.x & 31;
    __syncwarp();
    const longlong2 first = a.sipos[s0];
    float mx = 0.f, my = 0.f;
    bool nan_c = false;
    for (uint32_t i = lane; i < k; i += 32) {
        const longlong2 ip = a.sipos[s0 + i];
        const float c = a.sc[s0 + i];
        const float x = fx_to_f(ip.x - first.x), y = fx_to_f(ip.y - first.y);
        m.pos[i] = make_float2(x, y);
        m.cb[i] = make_float2(c, 0.f);
        m.id[i] = a.sorted[s0 + i];
        if (with_xy) m.xy[i] = a.sfpos[s0 + i];
        mx = fmaxf(mx, fabsf(x));
        my = fmaxf(my, fabsf(y));
        nan_c |= !(c == c);
    }
    /* non-negative floats order as their bits */
    o.Mx = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(mx)));
    o.My = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(my)));
    /* a member outside the frame's range: every pair of the leaf is exact */
    if (__any_sync(0xffffffffu, nan_c)) o.Mx = __int_as_float(0x7f800000);
    for (uint32_t i = lane; i < k; i += 32) m.cb[i].y = pair_band(a.f, m.cb[i].x, o.Mx, o.My);
    o.g = g;
    o.X0 = first.x;
    o.Y0 = first.y;
    __syncwarp();
}

/* q - r^2 in metres^2 */
__device__ inline float screen_q(const Frame &f, float dx, float dy, float c) {
    const float mx = dx * c, my = dy * f.cy;
    return __fmaf_rn(mx, mx, __fmaf_rn(my, my, -f.r2));
}

/* warp-collective: part `part` of `parts` of one work item (leaf g, chunk).  The
 * pairs of an item are numbered and dealt to the lanes of its warps 32 at a
 * time, so that every lane has a pair whatever the leaf's size; a lane steps its
 * pair along without a division. */
template <bool kFp64>
__device__ inline void refine_item(const RefineArgs &a, uint32_t g, uint32_t chunk, const LeafTile &m, LeafOrigin &o,
                                   RefineTally &t, uint32_t &qn, uint32_t tag, uint32_t part = 0,
                                   uint32_t parts = 1) {
    const int lane = threadIdx.x & 31;
    const uint32_t below = (1u << lane) - 1u;
    const Frame &f = a.f;
    const uint32_t s0 = a.grid_start[g];
    const uint32_t cnt_g = a.grid_count[g];
    const uint32_t k = cnt_g < a.cap ? cnt_g : a.cap;
    if (k == 0) return;
    if (g != o.g) stage_leaf(a, g, s0, k, m, o, !kFp64);

    /* inside checks: the pairs {i, i + s mod k}, s = 1 .. k / 2 (half of the
     * last s when k is even): each pair once; p1 = the lower rank */
    if (chunk == 0 && k > 1) {
        const uint32_t total = k * (k - 1) / 2;
        if (lane == 0 && part == 0) t.cand += total;
        uint32_t i = part * 32 + lane, s = 1;
        for (uint32_t e0 = part * 32; e0 < total; e0 += 32 * parts) {
            while (i >= k) {
                i -= k;
                ++s;
            }
            uint32_t j = i + s;
            if (j >= k) j -= k;
            const uint32_t lo = min(i, j), hi = max(i, j);
            bool hit = false;
            if (e0 + lane < total) {
                const float2 A = m.pos[lo], B = m.pos[hi], cb = m.cb[lo];
                const float d = screen_q(f, A.x - B.x, A.y - B.y, cb.x);
                if (kFp64) {
                    hit = !(d > cb.y);
                } else {
                    hit = d < 0.f;
                    if (!(fabsf(d) > cb.y)) {
                        ++t.band;
                        hit = pair_exact(a.sxy, s0 + lo, s0 + hi, a.ex);
                    }
                    t.hits += hit ? 1 : 0;
                }
            }
            const unsigned any = __ballot_sync(0xffffffffu, hit);
            if (any) {
                if (hit) {
                    QEntry &q = m.Q[qn + __popc(any & below)];
                    const uint32_t p1 = m.id[lo], p2 = m.id[hi];
                    q.pw = pair_word(p1, p2); /* ids ascend with rank */
                    q.prio = prio_pack(0, p1, 0, hi);
                    if (kFp64) {
                        q.v = make_uint4(s0 + lo, s0 + hi, 0, 0);
                    } else {
                        const float2 P = m.xy[lo], R = m.xy[hi];
                        q.v = make_uint4(__float_as_uint(P.x), __float_as_uint(P.y), __float_as_uint(R.x),
                                         __float_as_uint(R.y));
                    }
                }
                drain_if_full<kFp64>(a, m.Q, qn, __popc(any), tag, t);
            }
            i += 32 * parts;
        }
    }

    /* cross-leaf checks that target this leaf, this item's chunk: p1 = the
     * querier.  32 checks are loaded at once, one per lane (their chain of
     * dependent loads is paid once for the 32), and handed to the lanes that
     * test them by shuffles. */
    uint32_t tb, te;
    item_checks(a, g, chunk, tb, te);
    for (uint32_t t0 = tb; t0 < te; t0 += 32) {
        const uint32_t nc = te - t0 < 32 ? te - t0 : 32;
        uint32_t q = 0, ord = 0, qr = 0;
        float2 qf = make_float2(0.f, 0.f);
        float px = 0.f, py = 0.f, cq = 0.f, bq = 0.f;
        float lx = 0.f, ly = 0.f, hy = 0.f; /* the querier's own leaf */
        bool qstored = false;
        if ((uint32_t)lane < nc) {
            const uint2 qe = a.tlist[t0 + lane];
            q = qe.x;
            ord = qe.y;
            const uint2 rl = a.rank[q];
            qstored = !(rl.x & kDropped);
            qr = rl.x & ~kDropped;
            const IBox own = a.ibox[rl.y];
            const longlong2 qi = a.sipos[qr];
            cq = a.sc[qr];
            if (!kFp64) qf = a.sfpos[qr];
            px = fx_to_f(qi.x - o.X0);
            py = fx_to_f(qi.y - o.Y0);
            bq = pair_band(f, cq, fmaxf(o.Mx, fabsf(px)), fmaxf(o.My, fabsf(py)));
            /* the querier's leaf, widened by its rounding (two units and a
             * few u of the offsets) */
            const float ex = 4.f + 1e-6f * (o.Mx + fabsf(px)), ey = 4.f + 1e-6f * (o.My + fabsf(py));
            lx = fx_to_f(own.x - o.X0);
            ly = fx_to_f(own.y - o.Y0);
            hy = fx_to_f(own.w - o.Y0);
            lx += ex + 1e-6f * fabsf(lx);
            ly += ey + 1e-6f * fabsf(ly);
            hy += ey + 1e-6f * fabsf(hy);
        }
        const uint32_t total = nc * k;
        if (lane == 0 && part == 0) t.cand += total;
        uint32_t c = 0, j = part * 32 + lane; /* the lane's check (of the 32) and member */
        for (uint32_t e0 = part * 32; e0 < total; e0 += 32 * parts) {
            while (j >= k) {
                j -= k;
                ++c;
            }
            const float X = __shfl_sync(0xffffffffu, px, c), Y = __shfl_sync(0xffffffffu, py, c);
            const float C = __shfl_sync(0xffffffffu, cq, c), Bd = __shfl_sync(0xffffffffu, bq, c);
            bool hit = false;
            float2 P = make_float2(0.f, 0.f);
            const bool mine = e0 + lane < total;
            float d = 1.f;
            if (mine) {
                P = m.pos[j];
                d = screen_q(f, X - P.x, Y - P.y, C);
                hit = kFp64 ? !(d > Bd) : !(d > Bd) && !(d < -Bd) ? true : d < 0.f;
            }
            if (!__any_sync(0xffffffffu, hit)) {
                j += 32 * parts;
                continue;
            }
            const uint32_t Q0 = __shfl_sync(0xffffffffu, q, c), R0 = __shfl_sync(0xffffffffu, qr, c);
            const uint32_t O0 = __shfl_sync(0xffffffffu, ord, c);
            const bool st = __shfl_sync(0xffffffffu, (int)qstored, c) != 0;
            const float LX = __shfl_sync(0xffffffffu, lx, c), LY = __shfl_sync(0xffffffffu, ly, c);
            const float HY = __shfl_sync(0xffffffffu, hy, c);
            float2 F0 = make_float2(0.f, 0.f);
            if (!kFp64) {
                F0.x = __shfl_sync(0xffffffffu, qf.x, c);
                F0.y = __shfl_sync(0xffffffffu, qf.y, c);
            }
            uint32_t mm = 0;
            bool dup = false;
            if (hit) {
                mm = m.id[j];
                /* The pair is tested from mm's side too when mm has a check on
                 * q's leaf, which lies above mm, or level with it and to its
                 * right (the walk's rule, k_filter.cu): only then are mm's
                 * checks looked at. */
                dup = Q0 > mm && st && (!(P.y >= LY) || (!(P.x >= LX) && !(P.y >= HY)));
                if (!kFp64) {
                    if (!(fabsf(d) > Bd)) {
                        ++t.band;
                        hit = pair_exact(a.sxy, R0, s0 + j, a.ex);
                    }
                    t.hits += hit ? 1 : 0;
                    /* mm's test comes first in the reference's order when
                     * mm < q; keep only one event */
                    if (hit && dup && has_check(a, mm, a.info[R0].y)) {
                        const float cm = m.cb[j].x;
                        const float d2 = screen_q(f, P.x - X, P.y - Y, cm);
                        const float b2 = pair_band(f, cm, fmaxf(o.Mx, fabsf(X)), fmaxf(o.My, fabsf(Y)));
                        bool r2 = d2 < 0.f;
                        if (!(fabsf(d2) > b2)) {
                            ++t.band;
                            r2 = pair_exact(a.sxy, s0 + j, R0, a.ex);
                        }
                        if (r2) hit = false;
                    }
                }
            }
            const unsigned any = __ballot_sync(0xffffffffu, hit);
            if (any) {
                if (hit) {
                    QEntry &e = m.Q[qn + __popc(any & below)];
                    e.pw = pw_of(Q0, mm);
                    e.prio = prio_pack(1, Q0, O0, j);
                    if (kFp64) {
                        e.v = make_uint4(R0, s0 + j, dup ? 1u : 0u, 0u);
                    } else {
                        const float2 R = m.xy[j];
                        e.v = make_uint4(__float_as_uint(F0.x), __float_as_uint(F0.y), __float_as_uint(R.x),
                                         __float_as_uint(R.y));
                    }
                }
                drain_if_full<kFp64>(a, m.Q, qn, __popc(any), tag, t);
            }
            j += 32 * parts;
        }
    }
    __syncwarp();
}

/* warp-collective: this warp's share of one context's items.  Items are taken
 * from a cursor, except where there are no more of them than warps: then each
 * has its warp, or two or four when that many are left over, by number.  A small
 * region's few hundred items are otherwise one warp's chain of a whole leaf's
 * pairs each, behind two atomics: 2k objects 13.1 -> 7.0 us (FP32 screen), 20k
 * 16.1 -> 10.1 us (FP64).  From 100k objects on there are more items than warps. */
template <bool kFp64>
__device__ inline void refine_items(const RefineArgs &a, const LeafTile &m, RefineTally &t, uint32_t &qn,
                                    uint32_t tag) {
    const uint32_t nwork = a.cnt->n_leaf_work;
    const uint32_t n_extra = a.cnt->n_extra < a.extra_cap ? a.cnt->n_extra : a.extra_cap;
    const uint32_t items = nwork + n_extra, wpb = blockDim.x >> 5, warps = gridDim.x * wpb;
    LeafOrigin o;
    if (items <= warps) {
        const uint32_t parts = items * 4 <= warps ? 4u : items * 2 <= warps ? 2u : 1u;
        const uint32_t at = blockIdx.x * wpb + (threadIdx.x >> 5), v = at / parts;
        if (v >= items) return;
        const uint2 e = v < n_extra ? a.extra[v] : make_uint2(a.work[v - n_extra], 0u);
        refine_item<kFp64>(a, e.x, e.y, m, o, t, qn, tag, at - v * parts, parts);
        return;
    }
    bool extra_done = n_extra == 0;
    uint32_t g, chunk;
    while (claim_item(a, nwork, n_extra, extra_done, g, chunk)) refine_item<kFp64>(a, g, chunk, m, o, t, qn, tag);
}

/* warp-collective: the queued contacts into context a's table, and the
 * warp's counts into its totals */
template <bool kFp64>
__device__ inline void refine_flush(const RefineArgs &a, QEntry *Q, uint32_t &qn, uint32_t tag, RefineTally &t) {
    drain_queue<kFp64>(a, Q, qn, tag, t);
    qn = 0;
    for (int o = 16; o > 0; o >>= 1) {
        t.cand += __shfl_down_sync(0xffffffffu, t.cand, o);
        t.hits += __shfl_down_sync(0xffffffffu, t.hits, o);
        t.band += __shfl_down_sync(0xffffffffu, t.band, o);
    }
    if ((threadIdx.x & 31) == 0) {
        if (t.cand) atomicAdd(&a.cnt->candidates, t.cand);
        if (t.hits) atomicAdd(&a.cnt->contacts, t.hits);
        if (t.band) atomicAdd(&a.cnt->band_pairs, t.band);
    }
    t = RefineTally();
}

} // namespace glint

#endif
