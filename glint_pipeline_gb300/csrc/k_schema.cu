/*
 * k_schema.cu -- stage (a) part 2: split over-full leaves and merge
 * under-full quads, with the reference's one-step delay.
 *
 * Reference: update_schema_unit (tracing/filter.cpp:377-424) visits every
 * schema slot in index order.  A LEAF with width(true) > 2*reach and more than
 * grid_capacity objects counts an overflow and is split (split_node,
 * :338-375) once the count reaches schema_update_delay.  A BRANCH whose four
 * children are leaves holding fewer than grid_capacity objects together counts
 * an underflow and is merged (merge_node, :316-336).  Split pops four schema
 * slots and (after pushing the parent's grid) four grid ids from two stacks;
 * merge pushes the children back.  Because the pass runs in slot order, a
 * merge can make its parent's children all leaves before the parent is
 * visited (a cascade), and the slots and grid ids a split receives depend on
 * every earlier split and merge of the pass.
 *
 * Device form, same result:
 *  1. k_sch_collect: per slot, the split decision of each leaf and the merge
 *     decision of each branch whose children are all leaves; branches whose
 *     branch children all have smaller slots are merge candidates.
 *  2. k_sch_cascade: one block resolves the candidates bottom-up.
 *  3. events (split or merge) compacted in slot order by a scan.
 *  4. k_sch_apply: one block finds what each event takes from and leaves on
 *     the two stacks, and writes the node records.
 * Only the slots that have ever been in use (DevCounters::slots_used) are
 * looked at: the arrays hold 640,000 at least, whatever the region's size.
 */
#include "scan.cuh"

namespace glint {

enum : uint8_t { kEvNone = 0, kEvSplit = 1, kEvMerge = 2, kEvCand = 3, kEvFreed = 4 };

__global__ void __launch_bounds__(256) k_sch_collect(DNode *__restrict__ nodes, const double2 *__restrict__ low,
                                                     uint32_t S, const uint32_t *__restrict__ grid_count,
                                                     uint32_t gc, uint32_t delay, double two_r, ExactCtx ex,
                                                     uint8_t *__restrict__ flags, uint32_t *__restrict__ aux,
                                                     uint32_t *__restrict__ newgid, uint32_t *__restrict__ cand,
                                                     DevCounters *cnt) {
    if (cnt->slots_used && cnt->slots_used < S) S = cnt->slots_used;
    for (uint32_t s = blockIdx.x * blockDim.x + threadIdx.x; s < S; s += gridDim.x * blockDim.x) {
        const DNode n = nodes[s];
        uint8_t f = kEvNone;
        if (n.type == kLeaf) {
            const uint32_t c = grid_count[n.gid];
            bool cond = false;
            if (c > gc) {
                const double2 lo = low[s];
                cond = width_gt_exact(lo.x, kdbl(n.khx), lo.y, two_r, ex);
            }
            int16_t of = 0;
            if (cond) {
                of = (int16_t)(n.of + 1);
                if ((uint32_t)of >= delay) {
                    f = kEvSplit;
                    of = 0;
                }
            }
            if (of != n.of) nodes[s].of = of;
        } else if (n.type == kBranch) {
            bool ok = true, has_branch = false;
            uint32_t sum = 0;
            for (int i = 0; i < 4; ++i) {
                const uint32_t ch = n.child[i];
                const DNode cn = nodes[ch];
                if (cn.type == kLeaf) sum += grid_count[cn.gid];
                else if (cn.type == kBranch && ch < s) has_branch = true;
                else ok = false;
            }
            int16_t uf = 0;
            if (ok && !has_branch) {
                if (sum < gc) {
                    uf = (int16_t)(n.uf + 1);
                    if ((uint32_t)uf >= delay) {
                        f = kEvMerge;
                        uf = 0;
                        newgid[s] = nodes[n.child[3]].gid;
                    }
                }
                if (uf != n.uf) nodes[s].uf = uf;
            } else if (ok) {
                f = kEvCand;
                aux[s] = sum;
                uint32_t idx = atomicAdd(&cnt->n_cand, 1u);
                cand[idx] = s;
            } else if (n.uf != 0) {
                nodes[s].uf = 0;
            }
        }
        flags[s] = f;
    }
}

/* bottom-up resolution of merge candidates (branches with branch children of
 * smaller slot); at most tree-depth rounds */
__global__ void __launch_bounds__(1024) k_sch_cascade(DNode *__restrict__ nodes, uint8_t *__restrict__ flags,
                                                      const uint32_t *__restrict__ aux, uint32_t *__restrict__ newgid,
                                                      const uint32_t *__restrict__ cand, uint32_t gc, uint32_t delay,
                                                      DevCounters *cnt) {
    __shared__ int changed;
    const uint32_t nc = cnt->n_cand;
    for (int round = 0; round < 80; ++round) {
        if (threadIdx.x == 0) changed = 0;
        __syncthreads();
        for (uint32_t i = threadIdx.x; i < nc; i += blockDim.x) {
            const uint32_t g = cand[i];
            if ((flags[g] & 3) != kEvCand) continue;
            const DNode n = nodes[g];
            bool all_merge = true, resolved = true;
            for (int k = 0; k < 4; ++k) {
                const uint32_t ch = n.child[k];
                const uint8_t cf = flags[ch] & 3;
                if (nodes[ch].type != kBranch) continue;   /* a leaf child */
                if (cf == kEvMerge) continue;
                if (cf == kEvCand) resolved = false;
                else all_merge = false;
            }
            if (!all_merge) {
                flags[g] = kEvNone;
                if (n.uf != 0) nodes[g].uf = 0;
                changed = 1;
            } else if (resolved) {
                int16_t uf = 0;
                uint8_t f = kEvNone;
                if (aux[g] < gc) {
                    uf = (int16_t)(n.uf + 1);
                    if ((uint32_t)uf >= delay) {
                        f = kEvMerge;
                        uf = 0;
                        const uint32_t c3 = n.child[3];
                        newgid[g] = (flags[c3] & 3) == kEvMerge ? newgid[c3] : nodes[c3].gid;
                    }
                }
                if (uf != n.uf) nodes[g].uf = uf;
                __threadfence_block();
                flags[g] = f;
                changed = 1;
            }
        }
        __syncthreads();
        if (!changed) break;
    }
    /* anything still unresolved cannot merge */
    for (uint32_t i = threadIdx.x; i < nc; i += blockDim.x) {
        const uint32_t g = cand[i];
        if ((flags[g] & 3) == kEvCand) flags[g] = kEvNone;
    }
}

/* The events (splits and merges) in slot order: a scan whose values are made
 * from the flags as it loads them, and whose prefixes place the events.  On
 * the way the children of merged branches are marked as freed (a merged child
 * must not become a leaf again). */
struct EventIn {
    const DNode *nodes;
    uint8_t *flags;
    __device__ uint32_t at(uint32_t s) const {
        const uint8_t f = flags[s] & 3;
        return f == kEvMerge || f == kEvSplit ? 1u : 0u;
    }
    __device__ void load(uint32_t base, uint32_t n, uint32_t (&v)[kScanItems]) const {
#pragma unroll
        for (int k = 0; k < kScanItems; ++k) {
            const uint32_t s = base + k;
            v[k] = s < n ? at(s) : 0u;
            if (!v[k] || (flags[s] & 3) != kEvMerge) continue;
            for (int i = 0; i < 4; ++i) {
                const uint32_t ch = nodes[s].child[i];
                if ((flags[ch] & 3) == kEvMerge)
                    atomicOr(reinterpret_cast<unsigned int *>(flags + (ch & ~3u)),
                             (unsigned int)kEvFreed << (8 * (ch & 3u)));
            }
        }
    }
};
struct EventOut {
    uint32_t *events;
    DevCounters *cnt;
    __device__ void total(uint32_t, uint32_t sum) const { cnt->n_events = sum; }
    __device__ void store(uint32_t base, uint32_t, const uint32_t (&v)[kScanItems],
                          const uint32_t (&o)[kScanItems]) const {
#pragma unroll
        for (int k = 0; k < kScanItems; ++k)
            if (v[k]) events[o[k]] = base + k;
    }
};

/* ---- the events applied, in one block ----------------------------------------
 * The reference pops and pushes the two stacks event by event.  In terms of
 * the level (splits minus merges before an event) a split at level k pops
 * cell k, four schema slots and three grids, and a merge at level k pushes cell
 * k - 1 (and the grid below it, which the cell's own next merge or the stack
 * index hides).  Between two events that cross one cell the level returns to
 * it, so a split pops what the event that crossed its cell before it pushed,
 * which is a merge, or the stack's initial content.  So every event finds its
 * predecessor on its cell by itself: backwards among the 1024 events of its
 * round in shared memory, else in a table of each cell's last event; and a
 * merge that ends as its cell's last event is the stack's final content there.
 * One thread replaying the stacks in a shared-memory window took 63 us for a
 * 1M-object step's 420 events and 745 us for 5200, beside launches of their own
 * for what events carry and for the node records; this takes 37 and 316 us for
 * all of it, and the whole update 4 launches instead of 9. */
constexpr int kApplyThreads = 1024;

struct ApplyArgs {
    DNode *nodes;
    double2 *low;
    IBox *ibox;
    float4 *cbox;
    Frame fr;
    const uint8_t *flags;
    const uint32_t *newgid;
    const uint32_t *events;
    uint4 *evdata;             /* [2 E]: a merge's child slots and grids, a split's */
    int32_t *cell;             /* [E] the cell each event crosses */
    uint32_t *last;            /* [S] each cell's last event + 1, from the lowest cell on */
    uint32_t *sstack, *gstack;
    uint32_t S, G;
    uint32_t *grid_count;
    DevCounters *cnt;
};

__device__ inline void apply_merge(const ApplyArgs &a, uint32_t g, const uint4 ch, const uint4 cg) {
    /* merge_node zeroes the counters of the grids it frees (filter.cpp:331) */
    a.grid_count[cg.x] = 0;
    a.grid_count[cg.y] = 0;
    a.grid_count[cg.z] = 0;
    a.grid_count[cg.w] = 0;
    a.nodes[ch.x].type = kInvalid;
    a.nodes[ch.y].type = kInvalid;
    a.nodes[ch.z].type = kInvalid;
    a.nodes[ch.w].type = kInvalid;
    if (!(a.flags[g] & kEvFreed)) {
        a.nodes[g].type = kLeaf;
        a.nodes[g].gid = a.newgid[g];
    }
}

__device__ inline void apply_split(const ApplyArgs &a, uint32_t p, const uint4 cs, const uint4 gs) {
    /* split_node zeroes the counters of the children's grids (filter.cpp:359) */
    a.grid_count[gs.x] = 0;
    a.grid_count[gs.y] = 0;
    a.grid_count[gs.z] = 0;
    a.grid_count[gs.w] = 0;
    const DNode pn = a.nodes[p];
    const double2 pl = a.low[p];
    const double pmx = kdbl(pn.kmx), pmy = kdbl(pn.kmy);
    /* split_node (tracing/filter.cpp:347-370): children are the parent's
     * quadrants, offset by half the parent's extent; the boxes are also
     * kept in fixed point for the filter's screening */
    const double xhalf = __dsub_rn(pmx, pl.x);
    const double yhalf = __dsub_rn(pmy, pl.y);
    const uint32_t ch[4] = {cs.x, cs.y, cs.z, cs.w};
    const uint32_t gg[4] = {gs.x, gs.y, gs.z, gs.w};
    for (int k = 0; k < 4; ++k) {
        const double ox = (k % 2 == 1) ? xhalf : 0.0;
        const double oy = (k / 2 == 1) ? yhalf : 0.0;
        DNode c;
        const double lx = __dadd_rn(pl.x, ox);
        const double ly = __dadd_rn(pl.y, oy);
        const double hx = __dadd_rn(pmx, ox);
        const double hy = __dadd_rn(pmy, oy);
        c.khx = dkey(hx);
        c.khy = dkey(hy);
        c.kmx = dkey(__dmul_rn(__dadd_rn(lx, hx), 0.5));
        c.kmy = dkey(__dmul_rn(__dadd_rn(ly, hy), 0.5));
        const IBox box = fx_box(lx, ly, hx, hy, a.fr);
        a.ibox[ch[k]] = box;
        a.cbox[4 * (size_t)p + k] = f_box(box);
        c.child[0] = c.child[1] = c.child[2] = c.child[3] = 0;
        c.gid = gg[k];
        c.type = kLeaf;
        c.pad0 = 0;
        c.level = (int16_t)(pn.level + 1);
        c.of = 0;
        c.uf = 0;
        c.pad1 = 0;
        a.nodes[ch[k]] = c;
        a.low[ch[k]] = make_double2(lx, ly);
    }
    DNode q = pn;
    q.type = kBranch;
    q.child[0] = ch[0];
    q.child[1] = ch[1];
    q.child[2] = ch[2];
    q.child[3] = ch[3];
    a.nodes[p] = q;
}

__global__ void __launch_bounds__(kApplyThreads) k_sch_apply(ApplyArgs a) {
    __shared__ int32_t s_cell[kApplyThreads];
    __shared__ int32_t s_min, s_max, s_carry, s_merges;
    __shared__ int32_t s_ws[32];
    const uint32_t E = a.cnt->n_events;
    if (E == 0) return;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    if (threadIdx.x == 0) {
        s_min = 0;
        s_max = 0;
        s_carry = 0;
        s_merges = 0;
    }
    __syncthreads();
    /* 1. each event's cell and what it carries: for a merge its four children
     * and the grids they hold at that point of the pass, for a split the
     * parent's grid */
    for (uint32_t base = 0; base < E; base += kApplyThreads) {
        const uint32_t i = base + threadIdx.x;
        int32_t d = 0;
        if (i < E) {
            const uint32_t s = a.events[i];
            const DNode n = a.nodes[s];
            if ((a.flags[s] & 3) == kEvMerge) {
                d = -1;
                uint32_t cg[4];
                for (int k = 0; k < 4; ++k) {
                    const uint32_t ch = n.child[k];
                    cg[k] = (a.flags[ch] & 3) == kEvMerge ? a.newgid[ch] : a.nodes[ch].gid;
                }
                a.evdata[2 * i] = make_uint4(n.child[0], n.child[1], n.child[2], n.child[3]);
                a.evdata[2 * i + 1] = make_uint4(cg[0], cg[1], cg[2], cg[3]);
            } else {
                d = 1;
                a.evdata[2 * i + 1] = make_uint4(n.gid, 0, 0, 0);
            }
        }
        int32_t x = d; /* inclusive scan of the level's changes */
        for (int o = 1; o < 32; o <<= 1) {
            const int32_t y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31) s_ws[wid] = x;
        __syncthreads();
        if (wid == 0) {
            int32_t v = s_ws[lane];
            for (int o = 1; o < 32; o <<= 1) {
                const int32_t y = __shfl_up_sync(0xffffffffu, v, o);
                if (lane >= o) v += y;
            }
            s_ws[lane] = v;
        }
        __syncthreads();
        const int32_t before = s_carry + (wid ? s_ws[wid - 1] : 0) + x - d;
        if (i < E) {
            a.cell[i] = d > 0 ? before : before - 1;
            atomicMin(&s_min, before);
            atomicMax(&s_max, before);
            if (d < 0) atomicAdd(&s_merges, 1);
        }
        __syncthreads();
        if (threadIdx.x == 0) s_carry += s_ws[31];
        __syncthreads();
    }
    const int64_t ssi0 = a.cnt->ssi, gsi0 = a.cnt->gsi;
    const int64_t s_lo = ssi0 + 4 * (int64_t)s_min - 4, s_hi = ssi0 + 4 * (int64_t)s_max + 4;
    const int64_t g_lo = gsi0 + 3 * (int64_t)s_min - 4, g_hi = gsi0 + 3 * (int64_t)s_max + 3;
    const int32_t lo = s_min - 1, cells = s_max - lo + 1;
    if (s_lo < 0 || s_hi > (int64_t)a.S || g_lo < 0 || g_hi > (int64_t)a.G || (uint32_t)cells > a.S) {
        if (threadIdx.x == 0) {
            atomicOr(&a.cnt->error_flags, GLINT_EF_SCHEMA_STACK);
            a.cnt->n_events = 0; /* nothing is applied */
        }
        return;
    }
    for (int32_t i = threadIdx.x; i < cells; i += kApplyThreads) a.last[i] = 0;
    __syncthreads();
    /* 2. what each split pops */
    for (uint32_t base = 0; base < E; base += kApplyThreads) {
        const uint32_t i = base + threadIdx.x;
        const bool mine = i < E;
        const int32_t c = mine ? a.cell[i] : INT32_MIN;
        s_cell[threadIdx.x] = c;
        __syncthreads();
        if (mine && (a.flags[a.events[i]] & 3) == kEvSplit) {
            int j = (int)threadIdx.x - 1;
            while (j >= 0 && s_cell[j] != c) --j;
            const uint32_t from = j >= 0 ? base + j + 1 : a.last[c - lo];
            const uint32_t pg = a.evdata[2 * i + 1].x;
            uint4 cs, gs;
            if (from) {
                const uint4 ms = a.evdata[2 * (from - 1)], mg = a.evdata[2 * (from - 1) + 1];
                cs = make_uint4(ms.w, ms.z, ms.y, ms.x);
                gs = make_uint4(pg, mg.z, mg.y, mg.x);
            } else {
                const uint32_t *ss = a.sstack + ssi0 + 4 * (int64_t)c, *gr = a.gstack + gsi0 + 3 * (int64_t)c;
                cs = make_uint4(ss[0], ss[1], ss[2], ss[3]);
                gs = make_uint4(pg, gr[0], gr[1], gr[2]);
            }
            /* split_node (filter.cpp:343-358) */
            a.evdata[2 * i] = cs;
            a.evdata[2 * i + 1] = gs;
        }
        __syncthreads();
        if (mine) atomicMax(&a.last[c - lo], i + 1);
        __syncthreads();
    }
    /* 3. the stacks' final content (merge_node, filter.cpp:323-334), then the
     * node records: merges first */
    for (uint32_t i = threadIdx.x; i < E; i += kApplyThreads) {
        const uint32_t s = a.events[i];
        if ((a.flags[s] & 3) != kEvMerge) continue;
        const uint4 ms = a.evdata[2 * i], mg = a.evdata[2 * i + 1];
        const int32_t c = a.cell[i];
        if (a.last[c - lo] == i + 1) {
            uint32_t *ss = a.sstack + ssi0 + 4 * (int64_t)c, *gr = a.gstack + gsi0 + 3 * (int64_t)c;
            ss[0] = ms.w;
            ss[1] = ms.z;
            ss[2] = ms.y;
            ss[3] = ms.x;
            gr[0] = mg.z;
            gr[1] = mg.y;
            gr[2] = mg.x;
        }
        apply_merge(a, s, ms, mg);
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < E; i += kApplyThreads) {
        const uint32_t s = a.events[i];
        if ((a.flags[s] & 3) == kEvSplit) apply_split(a, s, a.evdata[2 * i], a.evdata[2 * i + 1]);
    }
    if (threadIdx.x == 0) {
        a.cnt->ssi = (unsigned)(ssi0 + 4 * (int64_t)s_carry);
        a.cnt->gsi = (unsigned)(gsi0 + 3 * (int64_t)s_carry);
        a.cnt->merges = (unsigned)s_merges;
        a.cnt->splits = E - (unsigned)s_merges;
        if (a.cnt->slots_used && a.cnt->slots_used < s_hi) a.cnt->slots_used = (unsigned)s_hi;
        if (a.cnt->grids_used && a.cnt->grids_used < g_hi) a.cnt->grids_used = (unsigned)g_hi;
    }
}

cudaError_t launch_schema_update(glint_ctx *c, cudaStream_t s, void *scan_tmp) {
    const uint32_t S = c->S;
    ExactCtx ex = make_exact(c);
    k_sch_collect<<<grid_for(S, 256, 152u * 8u), 256, 0, s>>>(c->d_nodes, c->d_low, S, c->d_grid_count,
                                                               c->cfg.grid_capacity, c->cfg.schema_update_delay,
                                                               2.0 * c->cfg.reach_distance, ex, c->d_split,
                                                               c->d_evscan, c->d_newgid, c->d_cand, c->d_cnt);
    k_sch_cascade<<<1, 1024, 0, s>>>(c->d_nodes, c->d_split, c->d_evscan, c->d_newgid, c->d_cand,
                                     c->cfg.grid_capacity, c->cfg.schema_update_delay, c->d_cnt);
    scan_launch(EventIn{c->d_nodes, c->d_split}, EventOut{c->d_evlist, c->d_cnt}, S, &c->d_cnt->slots_used, scan_tmp,
                s);
    ApplyArgs a;
    a.nodes = c->d_nodes;
    a.low = c->d_low;
    a.ibox = c->d_ibox;
    a.cbox = c->d_cbox;
    a.fr = c->frame;
    a.flags = c->d_split;
    a.newgid = c->d_newgid;
    a.events = c->d_evlist;
    a.evdata = c->d_evdata;
    a.cell = c->d_evlevel;
    a.last = c->d_evscan;
    a.sstack = c->d_sstack;
    a.gstack = c->d_gstack;
    a.S = S;
    a.G = c->G;
    a.grid_count = c->d_grid_count;
    a.cnt = c->d_cnt;
    k_sch_apply<<<1, kApplyThreads, 0, s>>>(a);
    return cudaGetLastError();
}

} // namespace glint
