/*
 * scan.cuh -- exclusive scan of 32-bit values in one launch, with the load
 * of the values and the use of their prefixes given by the caller, so that a
 * pass which makes the values or consumes their places is part of the scan.
 */
#ifndef GLINT_SCAN_CUH_
#define GLINT_SCAN_CUH_

#include <algorithm>

#include "glint_internal.cuh"

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

__device__ inline unsigned long long scan_status(uint32_t epoch, uint32_t flag, uint32_t value) {
    return ((unsigned long long)((epoch << 2) | flag) << 32) | value;
}

/* plain arrays: in[base ..], in whole 16-byte words when both are aligned */
struct ScanWords {
    const uint32_t *in;
    bool vec;
    __device__ uint32_t at(uint32_t i) const { return in[i]; }
    __device__ void load(uint32_t base, uint32_t n, uint32_t (&v)[kScanItems]) const {
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
    }
};

/* prefixes to out[0 .. n), their total to out[n] */
struct ScanStore {
    uint32_t *out;
    bool vec;
    __device__ void total(uint32_t n, uint32_t sum) const { out[n] = sum; }
    /* every thread of the block calls this, with its items from base on */
    __device__ void store(uint32_t base, uint32_t n, const uint32_t (&)[kScanItems],
                          const uint32_t (&o)[kScanItems]) const {
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
};

/* values [0, n), n = the lesser of n_max and *used (where used is given and
 * not zero): the launch covers n_max, tiles past n only sign off */
template <class In, class Out>
__global__ void __launch_bounds__(kScanThreads) k_scan(In in, Out out, uint32_t n_max,
                                                       const unsigned int *__restrict__ used, ScanHead *head) {
    constexpr uint32_t kSum = 1, kPrefix = 2;
    __shared__ uint32_t ws[kScanThreads / 32];
    __shared__ uint32_t s_tile, s_epoch, s_before;
    volatile unsigned long long *status = reinterpret_cast<unsigned long long *>(head + 1);
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    uint32_t n = n_max;
    if (used) {
        const uint32_t k = *used;
        if (k && k < n) n = k;
    }
    const uint32_t tiles = n ? (n + kScanTile - 1) / kScanTile : 1u;
    if (threadIdx.x == 0) {
        /* the epoch moves when the last block is done: all blocks read the same */
        s_epoch = (*(volatile uint32_t *)&head->epoch + 1) & 0x3fffffffu;
        s_tile = atomicAdd(&head->ticket, 1u);
    }
    __syncthreads();
    const uint32_t tile = s_tile, epoch = s_epoch;
    const uint32_t base = tile * kScanTile + threadIdx.x * kScanItems;
    uint32_t v[kScanItems];
    uint32_t mine = 0, incl = 0;
    if (tile < tiles) {
        in.load(base, n, v);
#pragma unroll
        for (int k = 0; k < kScanItems; ++k) mine += v[k];
        incl = mine;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += y;
        }
        if (lane == 31) ws[wid] = incl;
    }
    __syncthreads();
    if (wid == 0) {
        if (tile < tiles) {
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
                    for (uint32_t i = lane; i < tile * kScanTile; i += 32) before += in.at(i);
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
                if (tile == tiles - 1) out.total(n, before + sum);
            }
        }
        if (lane == 0 && atomicAdd(&head->done, 1u) == gridDim.x - 1) {
            head->ticket = 0;
            head->done = 0;
            head->epoch = epoch;
        }
    }
    __syncthreads();
    if (tile >= tiles) return;
    uint32_t p = s_before + ws[wid] + incl - mine;
    uint32_t o[kScanItems];
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) {
        o[k] = p;
        p += v[k];
    }
    out.store(base, n, v, o);
}

template <class In, class Out>
cudaError_t scan_launch(In in, Out out, uint32_t n_max, const unsigned int *used, void *tmp, cudaStream_t s) {
    const uint32_t tiles = std::max<uint32_t>(1, (n_max + kScanTile - 1) / kScanTile);
    k_scan<<<tiles, kScanThreads, 0, s>>>(in, out, n_max, used, (ScanHead *)tmp);
    return cudaGetLastError();
}

} // namespace glint

#endif
