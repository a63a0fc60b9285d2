/*
 * k_precision.cu -- the precision form of the refine stage: every candidate
 * pair is screened in FP32 on offsets from its leaf (refine_common.cuh), and
 * only the pairs whose screened squared distance lies inside the guard band
 * around r^2 are re-tested with the reference's FP64 arithmetic
 * (point_le_exact), so the contact set - and every meeting - stays identical
 * to the reference's.
 *
 * The reference's test (tracing/refinement.cpp:19-31 with Point::distance,
 * geometry/geometry.h:40-48) divides the longitude difference by L(y1) of the
 * checking object; the screen multiplies the offset difference by that
 * object's cx = 1/(L(y1) S).  No FP64 instruction runs per pair outside the
 * band: on sm_103a FP64 issues at a small fraction of the FP32 rate.
 *
 * Bound: issue slots at small tables, random record access at large ones.
 * Dealing pairs to lanes by number and loading 32 checks at a time took 1M
 * objects from 290 to 215 us, 2M in dense spots from 1562 to 1414 us and 10M
 * (34-GB table) from 10.4 to 9.5 ms.
 */
#include <algorithm>
#include <cstring>

#include <atomic>

#include "refine_common.cuh"

namespace glint {

constexpr int kPrecWarps = 4;

__global__ void __launch_bounds__(32 * kPrecWarps) k_refine_fp32(RefineArgs a) {
    extern __shared__ __align__(64) unsigned char smem_raw[];
    const LeafTile m = leaf_tile(smem_raw + (size_t)(threadIdx.x >> 5) * tile_warp_bytes(a.cap), a.cap);
    RefineTally t;
    uint32_t qn = 0;
    const uint32_t tag = a.cnt->step_tag;
    refine_items<false>(a, m, t, qn, tag);
    refine_flush<false>(a, m.Q, qn, tag, t);
}

/* ---- the refine stage of many contexts in one launch ---------------------
 * The items of all regions form one list: every region's extra chunks (the
 * long work) first, then every region's leaves.  A warp takes the next item,
 * finds its region, and works on it with that region's arguments, which it
 * keeps in its shared memory; before it moves to another region it drains
 * its queued contacts into the region it leaves.  Every contact carries its
 * place in the reference's order, so results do not depend on who tests it. */
/* one warp, 32 regions at a time: in one thread the counts are a chain of two
 * dependent loads a region (16 regions: 9.7 us, this way 2.6) */
__global__ void __launch_bounds__(32) k_refine_batch_prep(const RefineArgs *__restrict__ args, uint32_t R,
                                                          uint32_t *ex_off, uint32_t *wk_off, unsigned int *next) {
    const uint32_t lane = threadIdx.x;
    uint32_t e = 0, w = 0; /* the totals before these 32 */
    for (uint32_t r0 = 0; r0 < R; r0 += 32) {
        const uint32_t r = r0 + lane;
        uint32_t ne = 0, nw = 0;
        if (r < R) {
            const DevCounters *cnt = args[r].cnt;
            const uint64_t cap = args[r].extra_cap;
            nw = cnt->n_leaf_work;
            ne = cnt->n_extra;
            if (ne > cap) ne = (uint32_t)cap;
        }
        uint32_t pe = ne, pw = nw;
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t ue = __shfl_up_sync(0xffffffffu, pe, d), uw = __shfl_up_sync(0xffffffffu, pw, d);
            if (lane >= (uint32_t)d) {
                pe += ue;
                pw += uw;
            }
        }
        if (r < R) {
            ex_off[r] = e + pe - ne;
            wk_off[r] = w + pw - nw;
        }
        e += __shfl_sync(0xffffffffu, pe, 31);
        w += __shfl_sync(0xffffffffu, pw, 31);
    }
    if (lane == 0) {
        ex_off[R] = e;
        wk_off[R] = w;
        *next = 0;
    }
}

__device__ inline uint32_t region_of(const uint32_t *off, uint32_t R, uint32_t v) {
    uint32_t lo = 0, hi = R; /* off[lo] <= v < off[lo + 1] */
    while (hi - lo > 1) {
        const uint32_t mid = (lo + hi) / 2;
        if (off[mid] <= v) lo = mid;
        else hi = mid;
    }
    return lo;
}

__global__ void __launch_bounds__(32 * kPrecWarps) k_refine_fp32_batch(const RefineArgs *__restrict__ args, uint32_t R,
                                                                       const uint32_t *__restrict__ ex_off,
                                                                       const uint32_t *__restrict__ wk_off,
                                                                       unsigned int *next, uint32_t cap_max) {
    extern __shared__ __align__(64) unsigned char smem_raw[];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    constexpr size_t kArgBytes = (sizeof(RefineArgs) + 63) & ~(size_t)63;
    unsigned char *base = smem_raw + (size_t)w * (kArgBytes + tile_warp_bytes(cap_max));
    RefineArgs *sa = reinterpret_cast<RefineArgs *>(base);
    const LeafTile m = leaf_tile(base + kArgBytes, cap_max);
    const uint32_t E = ex_off[R], W = wk_off[R];
    RefineTally t;
    LeafOrigin o;
    uint32_t qn = 0, tag = 0, cur = ~0u;
    for (;;) {
        uint32_t v = 0;
        if (lane == 0) v = atomicAdd(next, 1u);
        v = __shfl_sync(0xffffffffu, v, 0);
        if (v >= E + W) break;
        uint32_t r, g, chunk;
        if (v < E) {
            r = region_of(ex_off, R, v);
            const uint2 e = args[r].extra[v - ex_off[r]];
            g = e.x;
            chunk = e.y;
        } else {
            r = region_of(wk_off, R, v - E);
            g = args[r].work[v - E - wk_off[r]];
            chunk = 0;
        }
        if (r != cur) {
            if (cur != ~0u) refine_flush<false>(*sa, m.Q, qn, tag, t);
            __syncwarp();
            static_assert(sizeof(RefineArgs) % 4 == 0, "RefineArgs words");
            const uint32_t *src = reinterpret_cast<const uint32_t *>(&args[r]);
            uint32_t *dst = reinterpret_cast<uint32_t *>(sa);
            for (uint32_t i = lane; i < sizeof(RefineArgs) / 4; i += 32) dst[i] = src[i];
            __syncwarp();
            cur = r;
            o.g = ~0u;
            tag = sa->cnt->step_tag;
        }
        refine_item<false>(*sa, g, chunk, m, o, t, qn, tag);
    }
    if (cur != ~0u) refine_flush<false>(*sa, m.Q, qn, tag, t);
}

int refine_prec_warps(uint32_t cap) {
    return (int)std::max<size_t>(1, std::min<size_t>(kPrecWarps, kMaxBlockSmem / tile_warp_bytes(cap)));
}

size_t refine_prec_smem_bytes(uint32_t cap) { return (size_t)refine_prec_warps(cap) * tile_warp_bytes(cap); }

cudaError_t launch_refine_precision(glint_ctx *c, const RefineArgs &a) {
    k_refine_fp32<<<152 * 8, 32 * refine_prec_warps(c->cap), refine_prec_smem_bytes(c->cap), c->stream>>>(a);
    return cudaGetLastError();
}

/* the refine pairs of R contexts in one launch on stream s; args, ex_off,
 * wk_off (R + 1 each) and next are device buffers of the caller */
cudaError_t launch_refine_precision_batch(const RefineArgs *d_args, uint32_t R, uint32_t cap_max, uint32_t *ex_off,
                                          uint32_t *wk_off, unsigned int *next, cudaStream_t s) {
    k_refine_batch_prep<<<1, 32, 0, s>>>(d_args, R, ex_off, wk_off, next);
    constexpr size_t kArgBytes = (sizeof(RefineArgs) + 63) & ~(size_t)63;
    const size_t per_warp = kArgBytes + tile_warp_bytes(cap_max);
    const int warps = (int)std::max<size_t>(1, std::min<size_t>(kPrecWarps, kMaxBlockSmem / per_warp));
    k_refine_fp32_batch<<<152 * 8, 32 * warps, warps * per_warp, s>>>(d_args, R, ex_off, wk_off, next, cap_max);
    return cudaGetLastError();
}

/* the per-kernel limit, set to the per-block maximum: every launch asks for
 * the shared memory its leaf buffer needs */
void refine_prec_set_attributes(uint32_t cap) {
    (void)cap;
    cudaFuncSetAttribute(k_refine_fp32, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMaxBlockSmem);
    cudaFuncSetAttribute(k_refine_fp32_batch, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMaxBlockSmem);
}

/* ---- probe: the screen against the FP64 test on sampled pairs --------------
 * Pairs (i, i + o), o = 1..32, for leaf-major ranks i = 0, stride, 2 stride,
 * ...: neighbours in that order share a leaf or sit in adjacent leaves, so the
 * sample is dominated by short distances, where the decision is made. */
struct ProbeAcc {
    unsigned long long pairs, in_band, mismatches, contacts;
    unsigned long long err_bits, err_near_bits, band_bits; /* non-negative doubles as bits */
};

__device__ inline unsigned long long warp_sum(unsigned long long v) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    return v;
}
__device__ inline unsigned long long warp_max(unsigned long long v) {
    for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long w = __shfl_down_sync(0xffffffffu, v, o);
        v = w > v ? w : v;
    }
    return v;
}

__global__ void __launch_bounds__(256) k_precision_probe(const longlong2 *__restrict__ sipos,
                                                         const double2 *__restrict__ sxy,
                                                         const float *__restrict__ sc, uint32_t N, uint32_t stride,
                                                         Frame f, ExactCtx ex, ProbeAcc *acc) {
    const unsigned long long samples = ((unsigned long long)N + stride - 1) / stride;
    const unsigned long long total = samples * 32;
    unsigned long long pairs = 0, band = 0, mism = 0, hits = 0;
    double err = 0.0, err_near = 0.0, bandm = 0.0;
    const double r = ex.r;
    const unsigned long long step = (unsigned long long)gridDim.x * blockDim.x;
    /* every lane runs the same number of iterations (the warp reductions
     * below need all 32) */
    const unsigned long long start = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x;
    for (unsigned long long it0 = start - (threadIdx.x & 31); it0 < total; it0 += step) {
        const unsigned long long it = it0 + (threadIdx.x & 31);
        const unsigned long long i = (it >> 5) * stride, j = i + (it & 31) + 1;
        if (it >= total || j >= N) continue;
        ++pairs;
        const longlong2 a = sipos[i], b = sipos[j];
        const float ci = sc[i], cj = sc[j];
        const long long dx = a.x - b.x, dy = a.y - b.y;
        const Screen s = make_screen(__fmaf_rn(0.0f, cj, ci), f);
        const int scr = fx_screen(dx, dy, s, f.cy);
        const double2 P = sxy[i], Q = sxy[j];
        const bool within = point_le_exact(P.x, P.y, Q.x, Q.y, dpm_lon_fast(P.y), ex);
        hits += within ? 1 : 0;
        if (scr < 0) ++band;
        else if ((scr == 1) != within) ++mism;
        const float mx = fx_to_f(dx) * s.cx, my = fx_to_f(dy) * f.cy;
        const float d32 = sqrtf(mx * mx + my * my);
        if (d32 == d32) {
            const double d64 = point_dist(P.x, P.y, Q.x, Q.y, dpm_lon_fast(P.y), ex.dpm_lat);
            const double e = fabs((double)d32 - d64);
            err = fmax(err, e);
            if (d64 <= 2.0 * r) err_near = fmax(err_near, e);
            const double bw = (double)(f.band0 + f.band1 * (s.cx + f.cy)) / (2.0 * r);
            if (bw == bw) bandm = fmax(bandm, bw);
        }
    }
    pairs = warp_sum(pairs);
    band = warp_sum(band);
    mism = warp_sum(mism);
    hits = warp_sum(hits);
    const unsigned long long eb = warp_max((unsigned long long)__double_as_longlong(err));
    const unsigned long long enb = warp_max((unsigned long long)__double_as_longlong(err_near));
    const unsigned long long bb = warp_max((unsigned long long)__double_as_longlong(bandm));
    if ((threadIdx.x & 31) == 0 && pairs) {
        atomicAdd(&acc->pairs, pairs);
        atomicAdd(&acc->in_band, band);
        atomicAdd(&acc->mismatches, mism);
        atomicAdd(&acc->contacts, hits);
        atomicMax(&acc->err_bits, eb);
        atomicMax(&acc->err_near_bits, enb);
        atomicMax(&acc->band_bits, bb);
    }
}

} // namespace glint

using namespace glint;

extern "C" glint_status glint_precision_probe(glint_ctx *c, uint32_t stride, glint_precision_report *out) {
    if (!c || !out || stride == 0) return GLINT_ERR_INVALID_ARGUMENT;
    if (c->step_index == 0) {
        c->last_error = "precision probe before the first step";
        return GLINT_ERR_STATE;
    }
    cudaSetDevice(c->device);
    ProbeAcc *d = nullptr;
    ProbeAcc h;
    std::memset(&h, 0, sizeof(h));
    cudaError_t e = cudaStreamSynchronize(c->stream);
    if (e == cudaSuccess) e = cudaMalloc((void **)&d, sizeof(ProbeAcc));
    if (e == cudaSuccess) e = cudaMemsetAsync(d, 0, sizeof(ProbeAcc), c->stream);
    if (e == cudaSuccess) {
        ExactCtx ex = make_exact(c);
        ex.ambiguous = nullptr; /* the step's counters stay the step's */
        ex.rechecks = nullptr;
        const unsigned long long total = (((unsigned long long)c->N + stride - 1) / stride) * 32;
        k_precision_probe<<<grid_for(total, 256, 152u * 8u), 256, 0, c->stream>>>(c->d_sipos, c->d_sxy, c->d_sc,
                                                                                 c->N, stride, c->frame, ex, d);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpyAsync(&h, d, sizeof(h), cudaMemcpyDeviceToHost, c->stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize(c->stream);
    if (d) cudaFree(d);
    if (e != cudaSuccess) {
        c->last_error = std::string("precision probe: ") + cudaGetErrorString(e);
        return e == cudaErrorMemoryAllocation ? GLINT_ERR_OUT_OF_MEMORY : GLINT_ERR_CUDA;
    }
    std::memset(out, 0, sizeof(*out));
    out->pairs = h.pairs;
    out->in_band = h.in_band;
    out->mismatches = h.mismatches;
    out->contacts = h.contacts;
    std::memcpy(&out->max_abs_err_m, &h.err_bits, sizeof(double));
    std::memcpy(&out->max_abs_err_near_m, &h.err_near_bits, sizeof(double));
    std::memcpy(&out->max_band_m, &h.band_bits, sizeof(double));
    out->stride = stride;
    return GLINT_OK;
}
