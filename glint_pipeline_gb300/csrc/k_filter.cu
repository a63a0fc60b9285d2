/*
 * k_filter.cu -- stage (b) part 1: cross-leaf checks for objects near the top
 * or right border of their leaf.
 *
 * Reference: filter_unit (tracing/filter.cpp:247-261) runs lookup_rec
 * (tracing/filter.cpp:130-152) from last_valid for every object whose
 * last_valid is not its own leaf: a depth-first walk over children 0..3 that
 * descends into branches within reach (box::distance, geometry/geometry.h:
 * 174-185) and keeps a leaf when it is within reach and lies above the
 * object, or level with and to its right.  Each kept leaf becomes a check
 * (object, leaf grid id, inside = false) appended after the N inside checks,
 * in object order and, per object, in walk order.
 *
 * Device form: one thread per border object, objects visited in leaf-major
 * order so that neighbouring threads walk the same nodes.  A node that comes off
 * the walk's stack is tested, kept or opened from words that are all requested
 * at once: its own, and its children's boxes in FP32, which rule out most of
 * the children; the others go on the stack in reverse order, so that they come
 * off in the reference's.  A node whose top is below the object is not opened:
 * nothing under it can be kept.  The walk reserves the object's place in the
 * check list and counts its checks by target leaf (which gives each its place
 * there) as it ends; after a scan of those counts the checks are copied, grouped
 * by target leaf, for the refine tiles.  The list by querier stays for the
 * duplicate rule in refine.
 *
 * Bound: the chain of dependent loads from node to child.  Testing one child at
 * a time, a load for its id and one for its words, took 125 us at 1M objects (29
 * us at 20k, for 3k border objects); four children at a time 105 (17.6), a node
 * in one load 92 (15.1).  10M: 1.72, 1.28 and 1.24 ms.
 */
#include <cmath>

#include "scan.cuh"

namespace glint {

constexpr int kQInline = 8;
/* 64 levels, each of which leaves at most three children waiting */
constexpr int kStackMax = 200;
constexpr uint32_t kWalkStart = 0x80000000u; /* the node a walk starts from is opened untested */

/* the querier of a walk: exact coordinates (for the top/right rule and the
 * exact fallback), fixed-point coordinates and screening limits */
struct WalkPoint {
    double px, py;
    long long X, Y;
    Screen sc;
    float fx, fy;        /* X, Y in FP32 */
    float rx, ry;        /* farther than this along an axis is out of reach, whatever FP32 rounded away */
    float top;           /* a box that ends below this ends below the object */
};

__device__ inline WalkPoint walk_point(const double2 p, const longlong2 ip, float c, const Frame &f) {
    WalkPoint w;
    w.px = p.x;
    w.py = p.y;
    w.X = ip.x;
    w.Y = ip.y;
    w.sc = make_screen(c, f);
    /* FP32 holds a coordinate to 2^-24 of itself (1.2 mm in a map of 40 km): a
     * gap of about the reach is off by less than 2^-22 of the coordinate and
     * two units */
    w.fx = fx_to_f(ip.x);
    w.fy = fx_to_f(ip.y);
    const float r = sqrtf(f.r2) * 1.0001f;
    const float ex = 4.f + 2.4e-7f * (fabsf(w.fx) + r / c), ey = 4.f + 2.4e-7f * (fabsf(w.fy) + r / f.cy);
    w.rx = r / c + ex;
    w.ry = r / f.cy + ey;
    w.top = w.fy - ey;
    return w;
}

/* the reference's FP64 box test for a box inside the guard band (rare); kept
 * out of line so that none of its FP64 work is scheduled on the common path */
__device__ __noinline__ bool box_exact(double lx, double ly, double hx, double hy, double px, double py,
                                       const ExactCtx &ex) {
    return box_le_exact(lx, ly, hx, hy, px, py, dpm_lon_fast(py), ex);
}

/* lookup_rec's walk of one object: the nodes and kept leaves still to visit,
 * in reverse order of the reference's depth-first walk */
struct Walk {
    uint32_t stack[kStackMax];
    int sp = 0;
    uint32_t kept = 0; /* leaves kept so far */
};

struct FilterArgs {
    const uint32_t *sorted;
    const double2 *sxy;
    const longlong2 *sipos;
    const float *sc;
    const uint2 *info;
    const DNode *nodes;
    const double2 *low;
    const IBox *ibox;
    const float4 *cbox;
    uint32_t N;
    Frame f;
    ExactCtx ex;
    DevCounters *cnt;
};

/* One step of a walk (of the start node only the children in `share` are
 * taken): the node on top is opened, or the kept leaf on top is
 * given to emit(gid, ordinal).  The box test is screened on the fixed-point
 * boxes; only a box within the guard band of the reach takes the reference's
 * FP64 box distance.  The top/right rule is decided on the fixed-point
 * coordinates where they are more than a unit apart, else on the doubles'
 * keys. */
template <class Emit>
__device__ inline void walk_step(const FilterArgs &a, Walk &k, const WalkPoint &w, uint32_t share, Emit emit) {
    const uint32_t e = k.stack[--k.sp], top = e & ~kWalkStart;
    const uint4 chv = *reinterpret_cast<const uint4 *>(a.nodes[top].child);
    const uint2 tail = *reinterpret_cast<const uint2 *>(&a.nodes[top].gid); /* gid; type, level */
    const IBox box = a.ibox[top];
    float4 fb[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) fb[i] = a.cbox[4 * (size_t)top + i];
    const uint32_t type = tail.y & 0xffu;
    if (!(e & kWalkStart)) {
        /* nothing at or above the object's latitude */
        if (box.w < w.Y - 1 && (type == kLeaf || type == kBranch)) return;
        int in = fx_box_screen(box, w.X, w.Y, w.sc, a.f.cy);
        if (in < 0) {
            atomicAdd(&a.cnt->box_band, 1u);
            const double2 lo = a.low[top];
            in = box_exact(lo.x, lo.y, kdbl(a.nodes[top].khx), kdbl(a.nodes[top].khy), w.px, w.py, a.ex) ? 1 : 0;
        }
        if (!in) return;
        if (type == kLeaf) {
            bool keep;
            if (w.Y < box.y - 1) {
                keep = true;
            } else if (w.Y > box.y + 1 && w.Y < box.w - 1 && (w.X < box.x - 1 || w.X > box.x + 1)) {
                keep = w.X < box.x;
            } else {
                const double2 lo = a.low[top];
                keep = dkey(w.py) < dkey(lo.y) || (dkey(w.py) < a.nodes[top].khy && dkey(w.px) < dkey(lo.x));
            }
            if (keep) emit(tail.x, k.kept++);
            return;
        }
        if (type != kBranch) {
            atomicOr(&a.cnt->error_flags, GLINT_EF_DFS_OVERFLOW);
            return;
        }
    }
    const uint32_t ch[4] = {chv.x, chv.y, chv.z, chv.w};
    if (!(e & kWalkStart)) share = 15u;
#pragma unroll
    for (int i = 3; i >= 0; --i) {
        if (!(share >> i & 1u) || fb[i].x - w.fx > w.rx || w.fx - fb[i].z > w.rx || fb[i].y - w.fy > w.ry || fb[i].w < w.top) continue;
        if (k.sp < kStackMax) k.stack[k.sp++] = ch[i];
        else atomicOr(&a.cnt->error_flags, GLINT_EF_DFS_OVERFLOW);
    }
}

/* Only border objects (a leaf beside their own in reach) walk the tree:
 * about half of them at 10M objects, a fifth at 1M.  Each warp reads 32
 * consecutive ranks at a time, queues its border objects in shared memory and
 * walks them 32 at a time, so that every lane of a walk has an object. */
constexpr int kWalkWarps = 4;
/* Maps of up to eight ranks for each of 24 warps an SM are read eight ranks at a
 * time, larger ones 32: a warp with at most eight border objects gives each four
 * lanes.  20k objects 15.1 -> 11.2 us, 2k 10.7 -> 8.0; read 16 at a time 100k
 * gained 1 us, and sixteen regions at once, which share the SMs, lost 2%. */
constexpr uint32_t kWalkSpread = 152 * 24;

struct CheckLists {
    uint32_t *qstart, *qcount; /* each object's checks */
    uint32_t *qlist;           /* their target leaves */
    uint32_t *qslot;           /* their places among their target's checks */
    uint32_t *tcount;          /* checks per target leaf */
    uint64_t cap;
};

__global__ void __launch_bounds__(32 * kWalkWarps) k_filter_walk(FilterArgs a, CheckLists l, uint32_t span) {
    __shared__ uint32_t sbuf[kWalkWarps][64];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const uint32_t below = (1u << lane) - 1u;
    const uint32_t stride = gridDim.x * kWalkWarps * span;
    uint32_t base = (blockIdx.x * kWalkWarps + wid) * span;
    uint32_t nb = 0, nborder = 0;
    for (;;) {
        while (nb < 32 && base < a.N) {
            const uint32_t i = base + lane;
            bool border = false;
            if (lane < (int)span && i < a.N) {
                border = a.info[i].x != kNoWalk;
                if (!border) l.qcount[a.sorted[i]] = 0;
            }
            const unsigned m = __ballot_sync(0xffffffffu, border);
            if (border) sbuf[wid][nb + __popc(m & below)] = i;
            nb += __popc(m);
            nborder += __popc(m);
            base += stride;
            __syncwarp();
        }
        if (nb == 0) break;
        /* the queue's last objects; of few, two or four lanes have one and
         * share the children of its start, in order */
        const uint32_t take = nb < 32 ? nb : 32;
        const uint32_t parts = take <= 8 ? 4u : take <= 16 ? 2u : 1u;
        const uint32_t obj = lane / parts, sub = lane % parts;
        const uint32_t share = parts == 4 ? 1u << sub : parts == 2 ? 3u << 2 * sub : 15u;
        const bool mine = obj < take;
        uint32_t pid = 0, lv = 0, row[kQInline];
        Walk k;
        WalkPoint w;
        if (mine) {
            const uint32_t i = sbuf[wid][nb - take + obj];
            pid = a.sorted[i];
            lv = a.info[i].x;
            w = walk_point(a.sxy[i], a.sipos[i], a.sc[i], a.f);
            k.sp = 1;
            k.stack[0] = lv | kWalkStart;
            while (k.sp > 0)
                walk_step(a, k, w, share, [&](uint32_t gid, uint32_t j) {
                    if (j < (uint32_t)kQInline) row[j] = gid;
                });
        }
        nb -= take;
        __syncwarp();
        /* the warp's checks take one run of the list */
        uint32_t n = k.kept, incl = n;
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += y;
        }
        const uint32_t head = lane - sub, tail = head + parts - 1;
        uint32_t at = 0;
        if (lane == 31 && incl) at = atomicAdd(&a.cnt->cross_checks, incl);
        at = __shfl_sync(0xffffffffu, at, 31) + incl - n;
        /* the object's run: from its first lane's to its last lane's end */
        const uint32_t from = __shfl_sync(0xffffffffu, at, head), to = __shfl_sync(0xffffffffu, at + n, tail);
        if (mine) {
            uint32_t all = to - from;
            if ((uint64_t)from + all > l.cap) {
                atomicOr(&a.cnt->error_flags, GLINT_EF_CHECKS_OVERFLOW);
                all = n = 0;
            }
            if (sub == 0) {
                l.qstart[pid] = from;
                l.qcount[pid] = all;
            }
            auto put = [&](uint32_t gid, uint32_t j) {
                l.qlist[at + j] = gid;
                l.qslot[at + j] = atomicAdd(&l.tcount[gid], 1u);
            };
            for (uint32_t j = 0; j < n && j < (uint32_t)kQInline; ++j) put(row[j], j);
            if (n > (uint32_t)kQInline) {
                /* the rare object with more: walked again for the rest */
                k.sp = 1;
                k.kept = 0;
                k.stack[0] = lv | kWalkStart;
                while (k.sp > 0)
                    walk_step(a, k, w, share, [&](uint32_t gid, uint32_t j) {
                        if (j >= (uint32_t)kQInline && j < n) put(gid, j);
                    });
            }
        }
        __syncwarp();
    }
    if (lane == 0 && nborder) atomicAdd(&a.cnt->border_objects, nborder);
}

/* group the checks by target leaf: tlist entries are (querier, ordinal) */
__global__ void __launch_bounds__(256) k_filter_group(uint32_t N, CheckLists l, const uint32_t *__restrict__ tstart,
                                                      uint2 *__restrict__ tlist) {
    for (uint32_t pid = blockIdx.x * blockDim.x + threadIdx.x; pid < N; pid += gridDim.x * blockDim.x) {
        const uint32_t n = l.qcount[pid];
        if (!n) continue;
        const uint32_t b = l.qstart[pid];
        for (uint32_t k = 0; k < n; ++k) tlist[tstart[l.qlist[b + k]] + l.qslot[b + k]] = make_uint2(pid, k);
    }
}

/* the scan of the checks per target leaf, and on the way the refine stage's
 * work items beyond each leaf's first (leaf, chunk of its checks) */
struct TargetScan {
    ScanStore start;
    const uint32_t *grid_count;
    uint2 *extra;
    uint64_t extra_cap;
    uint32_t per_item;
    DevCounters *cnt;
    __device__ void total(uint32_t n, uint32_t sum) const { start.total(n, sum); }
    __device__ void store(uint32_t base, uint32_t n, const uint32_t (&v)[kScanItems],
                          const uint32_t (&o)[kScanItems]) const {
        start.store(base, n, v, o);
#pragma unroll
        for (int k = 0; k < kScanItems; ++k) {
            if (v[k] <= per_item || !grid_count[base + k]) continue;
            const uint32_t chunks = (v[k] + per_item - 1) / per_item;
            const uint32_t at = atomicAdd(&cnt->n_extra, chunks - 1);
            for (uint32_t ch = 1; ch < chunks; ++ch) {
                if (at + ch - 1 < extra_cap) extra[at + ch - 1] = make_uint2(base + k, ch);
                else atomicOr(&cnt->error_flags, GLINT_EF_CHECKS_OVERFLOW);
            }
        }
    }
};

__global__ void __launch_bounds__(256) k_child_boxes(const DNode *__restrict__ nodes, const IBox *__restrict__ ibox,
                                                     uint32_t S, float4 *__restrict__ cbox) {
    for (uint32_t s = blockIdx.x * blockDim.x + threadIdx.x; s < S; s += gridDim.x * blockDim.x) {
        if (nodes[s].type != kBranch) continue;
        for (int i = 0; i < 4; ++i) {
            const uint32_t ch = nodes[s].child[i];
            if (ch < S) cbox[4 * (size_t)s + i] = f_box(ibox[ch]);
        }
    }
}

cudaError_t launch_child_boxes(glint_ctx *c) {
    k_child_boxes<<<grid_for(c->S, 256), 256, 0, c->stream>>>(c->d_nodes, c->d_ibox, c->S, c->d_cbox);
    return cudaGetLastError();
}

cudaError_t launch_filter(glint_ctx *c) {
    cudaStream_t s = c->stream;
    const uint32_t N = c->N, G = c->G;
    FilterArgs a;
    a.sorted = c->d_sorted;
    a.sxy = c->d_sxy;
    a.sipos = c->d_sipos;
    a.sc = c->d_sc;
    a.info = c->d_info;
    a.nodes = c->d_nodes;
    a.low = c->d_low;
    a.ibox = c->d_ibox;
    a.cbox = c->d_cbox;
    a.N = N;
    a.f = c->frame;
    a.ex = make_exact(c);
    a.cnt = c->d_cnt;
    CheckLists l;
    l.qstart = c->d_qstart;
    l.qcount = c->d_qcount;
    l.qlist = c->d_qlist;
    l.qslot = c->d_qslot;
    l.tcount = c->d_tcount;
    l.cap = c->check_cap;
    const uint32_t span = N <= 8 * kWalkSpread ? 8u : 32u;
    k_filter_walk<<<grid_for(N, span * kWalkWarps, 152u * 16u), 32 * kWalkWarps, 0, s>>>(a, l, span);
    TargetScan ts;
    ts.start = ScanStore{c->d_tstart, true};
    ts.grid_count = c->d_grid_count;
    ts.extra = c->d_rextra;
    ts.extra_cap = c->rextra_cap;
    ts.per_item = c->chunk;
    ts.cnt = c->d_cnt;
    scan_launch(ScanWords{c->d_tcount, true}, ts, G, &c->d_cnt->grids_used, c->d_scan_tmp, s);
    k_filter_group<<<grid_for(N, 256, 152u * 8u), 256, 0, s>>>(N, l, c->d_tstart, c->d_tlist);
    return cudaGetLastError();
}

} // namespace glint
