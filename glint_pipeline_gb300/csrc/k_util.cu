/*
 * k_util.cu -- device-wide exclusive scan, the double-double sin
 * coefficients, and the device side of the synthetic trajectory generator.
 */
#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <cstring>

#include "glint_internal.cuh"
#include "tracegen.h"

namespace glint {

/* Exclusive scan in one launch: a tile per block, the tiles' running sums
 * passed on by look-back over status words.  The step runs five scans, most
 * of them over a few hundred thousand words at most, so launches bound them:
 * the reduce / scan / down form took three (36 us for the five at 20k
 * objects), this takes one (26 us) and reads the input once instead of twice.
 * The scratch starts zeroed.  Its status words carry the scan's number
 * (epoch), so they need no reset between scans: a word of an earlier scan
 * reads as not there yet.  Tiles are taken by ticket, so a tile waits only for
 * tiles that already run; a wait that outlasts kScanPolls adds up the input
 * before its tile itself. */
constexpr int kScanThreads = 512;
constexpr int kScanItems = 8;
constexpr int kScanTile = kScanThreads * kScanItems;
constexpr uint32_t kScanPolls = 1u << 20;

struct ScanHead {
    uint32_t epoch, ticket, done, pad;
};

size_t scan_tmp_bytes(size_t n) {
    const size_t tiles = (n + kScanTile - 1) / kScanTile + 1;
    return sizeof(ScanHead) + tiles * sizeof(unsigned long long);
}

__device__ inline unsigned long long scan_status(uint32_t epoch, uint32_t flag, uint32_t value) {
    return ((unsigned long long)((epoch << 2) | flag) << 32) | value;
}

__global__ void __launch_bounds__(kScanThreads) k_scan(const uint32_t *__restrict__ in, uint32_t *__restrict__ out,
                                                       size_t n, ScanHead *head, uint32_t tiles, bool vec) {
    constexpr uint32_t kSum = 1, kPrefix = 2;
    __shared__ uint32_t ws[kScanThreads / 32];
    __shared__ uint32_t s_tile, s_epoch, s_before;
    volatile unsigned long long *status = reinterpret_cast<unsigned long long *>(head + 1);
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    if (threadIdx.x == 0) {
        /* the epoch moves when the last tile is done: all tiles read the same */
        s_epoch = (*(volatile uint32_t *)&head->epoch + 1) & 0x3fffffffu;
        s_tile = atomicAdd(&head->ticket, 1u);
    }
    __syncthreads();
    const uint32_t tile = s_tile, epoch = s_epoch;
    const size_t base = (size_t)tile * kScanTile + (size_t)threadIdx.x * kScanItems;
    uint32_t v[kScanItems];
    if (vec && base + kScanItems <= n) {
#pragma unroll
        for (int k = 0; k < kScanItems; k += 4) {
            const uint4 x = *reinterpret_cast<const uint4 *>(in + base + k);
            v[k] = x.x;
            v[k + 1] = x.y;
            v[k + 2] = x.z;
            v[k + 3] = x.w;
        }
    } else {
#pragma unroll
        for (int k = 0; k < kScanItems; ++k) v[k] = base + k < n ? in[base + k] : 0u;
    }
    uint32_t mine = 0;
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) mine += v[k];
    uint32_t incl = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
    }
    if (lane == 31) ws[wid] = incl;
    __syncthreads();
    if (wid == 0) {
        uint32_t w = lane < kScanThreads / 32 ? ws[lane] : 0u;
        const uint32_t own = w;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o) w += y;
        }
        const uint32_t sum = __shfl_sync(0xffffffffu, w, 31);
        if (lane < kScanThreads / 32) ws[lane] = w - own;
        if (lane == 0) status[tile] = scan_status(epoch, tile == 0 ? kPrefix : kSum, sum);
        uint32_t before = 0;
        for (long long at = (long long)tile - 1; at >= 0; at -= 32) {
            /* 32 earlier tiles at once, the nearest on lane 0 */
            const long long t = at - lane;
            unsigned long long st = scan_status(epoch, kPrefix, 0);
            uint32_t polls = 0;
            if (t >= 0) {
                do {
                    st = status[t];
                } while ((st >> 34) != epoch && ++polls < kScanPolls);
            }
            if (__any_sync(0xffffffffu, (st >> 34) != epoch)) {
                before = 0;
                for (size_t i = lane; i < (size_t)tile * kScanTile; i += 32) before += in[i];
                before = __reduce_add_sync(0xffffffffu, before);
                break;
            }
            const unsigned full = __ballot_sync(0xffffffffu, ((uint32_t)(st >> 32) & 3u) == kPrefix);
            const int upto = full ? __ffs(full) - 1 : 31;
            before += __reduce_add_sync(0xffffffffu, lane <= upto ? (uint32_t)st : 0u);
            if (full) break;
        }
        if (lane == 0) {
            if (tile) status[tile] = scan_status(epoch, kPrefix, before + sum);
            s_before = before;
            if (tile == tiles - 1) out[n] = before + sum;
            if (atomicAdd(&head->done, 1u) == tiles - 1) {
                head->ticket = 0;
                head->done = 0;
                head->epoch = epoch;
            }
        }
    }
    __syncthreads();
    uint32_t p = s_before + ws[wid] + incl - mine;
    uint32_t o[kScanItems];
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) {
        o[k] = p;
        p += v[k];
    }
    if (vec && base + kScanItems <= n) {
#pragma unroll
        for (int k = 0; k < kScanItems; k += 4)
            *reinterpret_cast<uint4 *>(out + base + k) = make_uint4(o[k], o[k + 1], o[k + 2], o[k + 3]);
    } else {
#pragma unroll
        for (int k = 0; k < kScanItems; ++k)
            if (base + k < n) out[base + k] = o[k];
    }
}

cudaError_t scan_u32(const uint32_t *in, uint32_t *out, size_t n, void *tmp, cudaStream_t s) {
    const uint32_t tiles = (uint32_t)std::max<size_t>(1, (n + kScanTile - 1) / kScanTile);
    const bool vec = (((uintptr_t)in | (uintptr_t)out) & 15) == 0;
    k_scan<<<tiles, kScanThreads, 0, s>>>(in, out, n, (ScanHead *)tmp, tiles, vec);
    return cudaGetLastError();
}

/* ---- double-double Taylor coefficients (-1)^k/(2k+1)!, computed on the host
 * in double-double with the same two-product/two-sum steps ---- */
static inline void h_quick(double a, double b, double &s, double &e) {
    s = a + b;
    e = b - (s - a);
}
static inline void h_div(double ah, double al, double d, double &qh, double &ql) {
    double q1 = ah / d;
    double p = q1 * d;
    double pe = std::fma(q1, d, -p);
    double r = ((ah - p) - pe) + al;
    double q2 = r / d;
    h_quick(q1, q2, qh, ql);
}

void init_sin_coef(SinCoef *c) {
    double fh = 1.0, fl = 0.0;
    c->hi[0] = 1.0;
    c->lo[0] = 0.0;
    for (int k = 1; k <= 20; ++k) {
        h_div(fh, fl, (double)(2 * k), fh, fl);
        h_div(fh, fl, (double)(2 * k + 1), fh, fl);
        c->hi[k] = (k & 1) ? -fh : fh;
        c->lo[k] = (k & 1) ? -fl : fl;
    }
}

} // namespace glint

/* ---- device trajectory generator ---- */
struct glint_gen {
    tg_params *d_params = nullptr;
    tg_object *d_objects = nullptr;
    uint32_t n = 0;
    uint32_t step = 0;    /* index of the next step produced */
};

__global__ void k_gen_step(const tg_params *__restrict__ P, tg_object *__restrict__ objs, uint32_t n, uint32_t step,
                           double *__restrict__ out) {
    const tg_params p = *P;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        tg_object o = objs[i];
        if (step > 0) tg_advance(&p, &o, i, step);
        double lon, lat;
        tg_position(&p, &o, &lon, &lat);
        objs[i] = o;
        reinterpret_cast<double2 *>(out)[i] = make_double2(lon, lat);
    }
}

extern "C" {

glint_status glint_gen_create(const void *params, uint32_t params_size, const void *objects, uint32_t num_objects,
                              uint32_t object_size, uint32_t first_step, glint_gen **out) {
    if (!params || !objects || !out || params_size != sizeof(tg_params) || object_size != sizeof(tg_object))
        return GLINT_ERR_INVALID_ARGUMENT;
    glint_gen *g = new glint_gen();
    g->n = num_objects;
    g->step = first_step;
    if (cudaMalloc(&g->d_params, sizeof(tg_params)) != cudaSuccess ||
        cudaMalloc(&g->d_objects, sizeof(tg_object) * (size_t)(num_objects ? num_objects : 1)) != cudaSuccess) {
        cudaFree(g->d_params);
        delete g;
        return GLINT_ERR_OUT_OF_MEMORY;
    }
    cudaMemcpy(g->d_params, params, sizeof(tg_params), cudaMemcpyHostToDevice);
    cudaMemcpy(g->d_objects, objects, sizeof(tg_object) * (size_t)num_objects, cudaMemcpyHostToDevice);
    *out = g;
    return cudaGetLastError() == cudaSuccess ? GLINT_OK : GLINT_ERR_CUDA;
}

glint_status glint_gen_step(glint_gen *g, double *d_out, void *stream) {
    if (!g || !d_out) return GLINT_ERR_INVALID_ARGUMENT;
    unsigned grid = glint::grid_for(g->n, 256, 152u * 16u);
    k_gen_step<<<grid, 256, 0, (cudaStream_t)stream>>>(g->d_params, g->d_objects, g->n, g->step, d_out);
    g->step++;
    return cudaGetLastError() == cudaSuccess ? GLINT_OK : GLINT_ERR_CUDA;
}

glint_status glint_gen_destroy(glint_gen *g) {
    if (!g) return GLINT_OK;
    cudaFree(g->d_params);
    cudaFree(g->d_objects);
    delete g;
    return GLINT_OK;
}

} /* extern "C" */
