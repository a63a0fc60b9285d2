/*
 * k_partition.cu -- stage (a): assign every object to its quadtree leaf and
 * lay the objects out leaf-major.
 *
 * Reference: the phased descent of filter_unit (tracing/filter.cpp:228-245)
 * and cuda_partition (cuda/geometry.cu:221-271): child = (y>mid_y)*2 +
 * (x>mid_x) from the root until a leaf, tracking last_valid, the deepest node
 * on the path whose top and right edges are more than x_buffer/y_buffer away.
 * workbench::insert (tracing/filter.cpp:95-111) then appends the object to
 * its leaf buffer and drops it once the buffer holds grid_capacity*amplify
 * objects; with one thread objects arrive in id order, so a leaf's stored
 * members are its smallest ids.
 *
 * Here the leaf buffers are replaced by a stable sort of objects by
 * (grid id, object id): a count per grid, which gives every object a place in
 * its grid's segment, an exclusive scan, a scatter and a per-leaf sort of each
 * segment, which also gathers what the later stages read in that order.  The first min(count, capacity) entries of a
 * segment are exactly the reference's stored members, in the same order.
 */
#include "scan.cuh"

namespace glint {

constexpr int kMaxDepth = 64;

__global__ void __launch_bounds__(256) k_descend(const double2 *const *in, const uint32_t *__restrict__ order,
                                                 uint32_t N, const DNode *__restrict__ nodes, uint32_t S, uint32_t G,
                                                 double xb, double yb, uint4 *__restrict__ obj,
                                                 uint32_t *__restrict__ grid_node,
                                                 uint32_t *__restrict__ grid_count, DevCounters *cnt) {
    const double2 *__restrict__ pts = *in;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < N; i += gridDim.x * blockDim.x) {
        const uint32_t pid = order[i];
        const double2 p = pts[pid];
        /* the comparisons of filter.cpp:231,235-236 on order-preserving keys */
        const uint64_t kx = dkey(p.x), ky = dkey(p.y);
        const uint64_t kxb = dkey(__dadd_rn(p.x, xb)), kyb = dkey(__dadd_rn(p.y, yb));
        uint32_t cur = 0, lv = 0, gid = 0;
        DNode n = nodes[0];
        int depth = 0;
        for (;;) {
            const int child = (ky > n.kmy) * 2 + (kx > n.kmx);
            cur = n.child[child];
            if (cur >= S || ++depth >= kMaxDepth) {
                /* a corrupt or too deep schema: keep memory safe and report */
                atomicOr(&cnt->error_flags, GLINT_EF_TREE_DEPTH);
                cur = lv = gid = 0;
                break;
            }
            n = nodes[cur];
            if (kxb < n.khx && kyb < n.khy) lv = cur;
            if (n.type == kLeaf) {
                gid = n.gid < G ? n.gid : 0u;
                break;
            }
            if (n.type != kBranch) {
                atomicOr(&cnt->error_flags, GLINT_EF_TREE_DEPTH);
                cur = lv = gid = 0;
                break;
            }
        }
        /* objects come in the previous step's leaf order, so the lanes of a
         * warp mostly share a leaf: one atomic per leaf and warp, which also
         * gives each object its place in the leaf's segment */
        const unsigned peers = __match_any_sync(__activemask(), gid);
        const int leader = __ffs(peers) - 1;
        uint32_t at = 0;
        if ((threadIdx.x & 31) == leader) at = atomicAdd(&grid_count[gid], (uint32_t)__popc(peers));
        at = __shfl_sync(peers, at, leader);
        at += __popc(peers & ((1u << (threadIdx.x & 31)) - 1u));
        if (at == 0) grid_node[gid] = cur;
        /* in the order of the launch, which is nearly the order that follows: by
         * object id this store, the scatter's and the walk's loads were a sector
         * an object each.  Descent, scatter and walk at 1M objects 48 + 10.3 + 93
         * us, so 46 + 3.7 + 91; at 10M 0.65 + 0.11 + 1.28 ms, 0.54 + 0.04 + 1.16 */
        obj[i] = make_uint4(pid, gid, lv == cur ? kNoWalk : lv, at);
    }
}

__global__ void __launch_bounds__(256) k_scatter(const uint4 *__restrict__ obj, uint32_t N,
                                                 const uint32_t *__restrict__ grid_start,
                                                 uint2 *__restrict__ unsorted) {
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < N; i += gridDim.x * blockDim.x) {
        const uint4 o = obj[i];
        unsorted[grid_start[o.y] + o.w] = make_uint2(o.x, o.z);
    }
}

/* the scan of the leaf counts: segment starts, and on the way the leaves that
 * hold objects (work, in any order), those whose segment is too long for one
 * warp (big) and the objects that their buffers drop */
struct LeafScan {
    ScanStore start;
    uint32_t *work, *big;
    uint32_t cap, warp_limit;
    DevCounters *cnt;
    __device__ void total(uint32_t n, uint32_t sum) const { start.total(n, sum); }
    __device__ void store(uint32_t base, uint32_t n, const uint32_t (&v)[kScanItems],
                          const uint32_t (&o)[kScanItems]) const {
        start.store(base, n, v, o);
        const int lane = threadIdx.x & 31;
        uint32_t have = 0, drop = 0;
#pragma unroll
        for (int k = 0; k < kScanItems; ++k) {
            have += v[k] ? 1u : 0u;
            drop += v[k] > cap ? v[k] - cap : 0u;
        }
        uint32_t incl = have;
        for (int s = 1; s < 32; s <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, incl, s);
            if (lane >= s) incl += y;
        }
        uint32_t at = 0;
        if (lane == 31 && incl) at = atomicAdd(&cnt->n_leaf_work, incl);
        at = __shfl_sync(0xffffffffu, at, 31) + incl - have;
#pragma unroll
        for (int k = 0; k < kScanItems; ++k) {
            if (!v[k]) continue;
            work[at++] = base + k;
            if (v[k] > warp_limit) big[atomicAdd(&cnt->n_big, 1u)] = base + k;
        }
        drop = __reduce_add_sync(0xffffffffu, drop);
        if (lane == 0 && drop) atomicAdd(&cnt->dropped, drop);
    }
};

/* per object, in leaf-major order: the coordinates, their fixed-point and
 * FP32 forms and the screening scale cx; metres per degree of longitude in
 * FP64 for the plain form; each object's sorted position */
struct GatherOut {
    double2 *sxy;
    longlong2 *sipos;
    float2 *sfpos;
    float *sc;
    double *sm;        /* null: not needed */
    float2 *fpos;      /* by object id */
    uint2 *rank;       /* by object id: sorted position and leaf node */
    uint32_t *sorted;
    uint2 *info;
    const uint2 *unsorted;     /* object and walk start, by leaf */
    const uint32_t *grid_node;
    uint32_t cap;
};

/* a segment: the leaf grid and node, and where it starts */
struct Segment {
    uint32_t g, leaf, s0;
};

/* object v (id and walk start) at place `at` of a segment */
__device__ inline void gather_one(const GatherOut &o, const Frame &f, const double2 p, const Segment &s, uint32_t at,
                                  const uint2 v) {
    const uint32_t i = s.s0 + at, pid = v.x;
    o.sorted[i] = pid;
    o.info[i] = make_uint2(v.y, s.g);
    o.sxy[i] = p;
    bool clamped = false;
    const long long X = fx_coord(p.x, f.k, f.X0, &clamped);
    const long long Y = fx_coord(p.y, f.k, f.Y0, &clamped);
    o.sipos[i] = make_longlong2(X, Y);
    o.sc[i] = clamped ? __int_as_float(0x7fc00000) : c_of_lat(p.y, f);
    const float2 fp = make_float2(f_of_d(p.x), f_of_d(p.y));
    o.sfpos[i] = fp;
    o.fpos[pid] = fp;
    if (o.sm) o.sm[i] = metres_per_degree(p.y, f);
    o.rank[pid] = make_uint2(at < o.cap ? i : i | kDropped, s.leaf);
}

/* A warp's segment of up to 32 K different ids: each lane counts the ids below
 * its own, which is their place.  One pass over the ids in shared memory, read
 * four at a time by all lanes at once, with the points' loads in flight behind
 * it; a bitonic network of the same segment is 15 to 28 stages, each waiting
 * for the one before. */
template <int K>
__device__ inline void rank_sort(const GatherOut &o, const Frame &f, const double2 *__restrict__ pts,
                                 uint32_t *buf, uint32_t n, const Segment &s) {
    const uint32_t lane = threadIdx.x & 31;
    uint2 v[K];
    uint32_t r[K];
    double2 p[K];
#pragma unroll
    for (int e = 0; e < K; ++e) {
        const uint32_t i = lane + 32 * e;
        v[e] = i < n ? o.unsorted[s.s0 + i] : make_uint2(0xffffffffu, 0u);
        buf[i] = v[e].x;
        r[e] = 0;
    }
#pragma unroll
    for (int e = 0; e < K; ++e)
        if (lane + 32 * e < n) p[e] = pts[v[e].x];
    __syncwarp();
    for (uint32_t j = 0; j < n; j += 4) {
        const uint4 q = *reinterpret_cast<const uint4 *>(buf + j);
#pragma unroll
        for (int e = 0; e < K; ++e) r[e] += (q.x < v[e].x) + (q.y < v[e].x) + (q.z < v[e].x) + (q.w < v[e].x);
    }
#pragma unroll
    for (int e = 0; e < K; ++e)
        if (lane + 32 * e < n) gather_one(o, f, p[e], s, r[e], v[e]);
}

constexpr int kSortWarps = 8;
constexpr uint32_t kWarpSortMax = 128;
constexpr uint32_t kRankSortMax = 512;

/* One warp per leaf segment of up to kWarpSortMax objects: its ids in order,
 * and each object's gathered arrays while the ids are still at hand.  Bound:
 * the scattered reads and writes by object id (about 100 bytes an object in
 * 32-byte sectors), and at small maps the chain of dependent loads from the
 * leaf to the point.  With a bitonic network: 1M objects 53 us, 20k 9.3, 2k
 * 8.3; ranked by counting: 37, 5.9 and 4.6.  Segments up to 1024 a warp left
 * 2M objects in dense spots waiting for a few warps: 249 us, 225 with the
 * counting alone; from 129 on by whole blocks 84 (and 47 in the block kernel,
 * 13 before; the line at 256: 115 and 36). */
__global__ void __launch_bounds__(32 * kSortWarps) k_segsort_warp(const uint32_t *__restrict__ work,
                                                                  const uint32_t *__restrict__ grid_start,
                                                                  const uint32_t *__restrict__ grid_count,
                                                                  const double2 *const *in, GatherOut o,
                                                                  Frame f, const DevCounters *cnt) {
    __shared__ __align__(16) uint32_t buf[kSortWarps][kWarpSortMax];
    const double2 *__restrict__ pts = *in;
    const int w = threadIdx.x >> 5;
    const uint32_t nwork = cnt->n_leaf_work;
    for (uint32_t li = blockIdx.x * kSortWarps + w; li < nwork; li += gridDim.x * kSortWarps) {
        const uint32_t g = work[li];
        const uint32_t n = grid_count[g];
        if (n > kWarpSortMax) continue;
        const Segment s = {g, o.grid_node[g], grid_start[g]};
        if (n <= 32) rank_sort<1>(o, f, pts, buf[w], n, s);
        else if (n <= 64) rank_sort<2>(o, f, pts, buf[w], n, s);
        else rank_sort<4>(o, f, pts, buf[w], n, s);
        __syncwarp();
    }
}

constexpr uint32_t kBlockSortMax = 16384;

/* One block per longer segment (up to kBlockSortMax objects): ranked by
 * counting up to kRankSortMax, with two or four threads an object, above that
 * by a bitonic network (counting grows with the square of the length: the line
 * at 1024 took 56 us where this takes 47, 2M objects in dense spots). */
__global__ void __launch_bounds__(1024) k_segsort_block(const uint32_t *__restrict__ big,
                                                        const uint32_t *__restrict__ grid_start,
                                                        const uint32_t *__restrict__ grid_count,
                                                        const double2 *const *in, GatherOut o, Frame f,
                                                        DevCounters *cnt) {
    extern __shared__ __align__(16) uint32_t sbuf[];
    const double2 *__restrict__ pts = *in;
    const uint32_t nbig = cnt->n_big;
    for (uint32_t bi = blockIdx.x; bi < nbig; bi += gridDim.x) {
        const uint32_t g = big[bi];
        const uint32_t n = grid_count[g];
        const Segment s = {g, o.grid_node[g], grid_start[g]};
        const uint2 *seg = o.unsorted + s.s0;
        if (n > kBlockSortMax) {
            /* reported; the arrays are filled all the same, so that what
             * follows in this step reads objects */
            if (threadIdx.x == 0) atomicOr(&cnt->error_flags, GLINT_EF_SEGMENT_TOO_LARGE);
            for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) gather_one(o, f, pts[seg[i].x], s, i, seg[i]);
            continue;
        }
        __syncthreads();
        if (n <= kRankSortMax) {
            const uint32_t parts = n <= kRankSortMax / 2 ? 4 : 2;
            const uint32_t i = threadIdx.x / parts, part = threadIdx.x % parts;
            if (threadIdx.x < kRankSortMax) sbuf[threadIdx.x] = threadIdx.x < n ? seg[threadIdx.x].x : 0xffffffffu;
            const uint2 me = i < n ? seg[i] : make_uint2(0u, 0u);
            const uint32_t v = me.x;
            double2 p = make_double2(0., 0.);
            if (i < n) p = pts[v];
            __syncthreads();
            uint32_t r = 0;
            for (uint32_t j = 4 * part; j < n; j += 4 * parts) {
                const uint4 q = *reinterpret_cast<const uint4 *>(sbuf + j);
                r += (q.x < v) + (q.y < v) + (q.z < v) + (q.w < v);
            }
            for (uint32_t d = 1; d < parts; d <<= 1) r += __shfl_xor_sync(0xffffffffu, r, d);
            if (i < n && part == 0) gather_one(o, f, p, s, r, me);
            continue;
        }
        uint32_t P = 1024;
        while (P < n) P <<= 1;
        for (uint32_t i = threadIdx.x; i < P; i += blockDim.x) sbuf[i] = i < n ? seg[i].x : 0xffffffffu;
        __syncthreads();
        for (uint32_t k = 2; k <= P; k <<= 1) {
            for (uint32_t j = k >> 1; j > 0; j >>= 1) {
                for (uint32_t i = threadIdx.x; i < P; i += blockDim.x) {
                    uint32_t l = i ^ j;
                    if (l > i) {
                        uint32_t a = sbuf[i], b = sbuf[l];
                        bool up = (i & k) == 0;
                        if ((a > b) == up) { sbuf[i] = b; sbuf[l] = a; }
                    }
                }
                __syncthreads();
            }
        }
        for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) {
            const uint2 v = seg[i];
            uint32_t lo = 0, hi = n; /* v's place: sbuf[lo] <= v < sbuf[hi] */
            while (hi - lo > 1) {
                const uint32_t mid = (lo + hi) / 2;
                if (sbuf[mid] <= v.x) lo = mid;
                else hi = mid;
            }
            gather_one(o, f, pts[v.x], s, lo, v);
        }
        __syncthreads();
    }
}

/* the start of a step: its counters cleared, its parameters taken in (by
 * value; from host memory in a batch's captured step), and the counts of the
 * leaves in use cleared */
__global__ void __launch_bounds__(256) k_step_begin(StepInput input, const StepInput *from, const double2 **in,
                                                    uint32_t *__restrict__ grid_count, uint32_t *__restrict__ tcount,
                                                    uint32_t G, DevCounters *cnt) {
    const uint32_t n = cnt->grids_used && cnt->grids_used < G ? cnt->grids_used : G;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        grid_count[i] = 0;
        tcount[i] = 0;
    }
    if (blockIdx.x == 0) {
        uint32_t *w = reinterpret_cast<uint32_t *>(cnt);
        for (uint32_t i = threadIdx.x; i < kStepCounterBytes / 4; i += blockDim.x) w[i] = 0;
        if (threadIdx.x == 0) {
            if (from) input = *from;
            *reinterpret_cast<StepParams *>(&cnt->step_time) = input.p;
            *in = input.pts;
        }
    }
}

cudaError_t launch_step_begin(glint_ctx *c, bool from_host) {
    k_step_begin<<<grid_for(c->G, 256, 152u * 4u), 256, 0, c->stream>>>(
        *c->h_input, from_host ? c->h_input : nullptr, c->d_in, c->d_grid_count, c->d_tcount, c->G, c->d_cnt);
    return cudaGetLastError();
}

cudaError_t launch_partition(glint_ctx *c) {
    cudaStream_t s = c->stream;
    const uint32_t N = c->N, G = c->G;
    /* the last step's leaf-major order is the descent's processing order */
    k_descend<<<grid_for(N, 256, 152u * 8u), 256, 0, s>>>(c->d_in, c->d_sorted, N, c->d_nodes, c->S, G, c->x_buffer,
                                                           c->y_buffer, c->d_obj, c->d_grid_node, c->d_grid_count,
                                                           c->d_cnt);
    LeafScan ls;
    ls.start = ScanStore{c->d_grid_start, true};
    ls.work = c->d_leaf_work;
    ls.big = c->d_big;
    ls.cap = c->cap;
    ls.warp_limit = kWarpSortMax;
    ls.cnt = c->d_cnt;
    scan_launch(ScanWords{c->d_grid_count, true}, ls, G, &c->d_cnt->grids_used, c->d_scan_tmp, s);
    k_scatter<<<grid_for(N, 256, 152u * 8u), 256, 0, s>>>(c->d_obj, N, c->d_grid_start, c->d_seg);
    GatherOut o;
    o.sxy = c->d_sxy;
    o.sipos = c->d_sipos;
    o.sfpos = c->d_sfpos;
    o.sc = c->d_sc;
    o.sm = c->cfg.precision_mode == 1 ? nullptr : c->d_sm;
    o.fpos = c->d_fpos;
    o.rank = c->d_rank;
    o.sorted = c->d_sorted;
    o.info = c->d_info;
    o.unsorted = c->d_seg;
    o.grid_node = c->d_grid_node;
    o.cap = c->cap;
    k_segsort_warp<<<grid_for(N, 16 * kSortWarps, 152u * 8u), 32 * kSortWarps, 0, s>>>(
        c->d_leaf_work, c->d_grid_start, c->d_grid_count, c->d_in, o, c->frame, c->d_cnt);
    k_segsort_block<<<304, 1024, kBlockSortMax * sizeof(uint32_t), s>>>(
        c->d_big, c->d_grid_start, c->d_grid_count, c->d_in, o, c->frame, c->d_cnt);
    return cudaGetLastError();
}

void partition_set_attributes() {
    cudaFuncSetAttribute(k_segsort_block, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)(kBlockSortMax * sizeof(uint32_t)));
}

} // namespace glint
