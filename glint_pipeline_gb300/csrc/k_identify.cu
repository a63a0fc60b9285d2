/*
 * k_identify.cu -- stage (d) part 2: expire finished meetings and emit the
 * ones that lasted long enough.
 *
 * Reference: update_meetings_unit (tracing/meeting.cpp:32-76) scans every
 * bucket: an entry touched this step (end == cur_time) is active; any other
 * entry is removed, and reported first when cur_time - start >=
 * min_meet_time + 1.  With one thread the reports come out in bucket order
 * (batch_meet, tracing/meeting.cpp:11-24).
 *
 * Device form: a stamp byte per bucket says empty or committed, and a bit per
 * 128-byte line of the table says that the insert placed a pair in it this
 * step, so the scan reads one byte per bucket and the 32-byte records only of
 * committed entries and of lines that received a pair.  Pass 1 finalises
 * entries inserted this step, removes expired entries that are too short,
 * marks the ones to report and counts them per tile; an exclusive scan gives
 * every tile its offset; pass 2 visits only tiles with reports and writes them
 * in bucket order into the device meeting log, then removes those entries.
 *
 * Bound: DRAM latency at the load factors in use (5-35%), where most lanes
 * that walk the buckets in order have nothing to read.  Each warp therefore
 * first lists the buckets of its span that need their record (pass 1) or hold
 * a report (pass 2) in shared memory, and then works through the list with
 * every lane busy and kIdIlp records per lane in flight.  Stamps are changed
 * in shared memory and written back as whole 16-byte words.  Walking in order
 * took 9.0 + 0.85 ms (pass 1 + pass 2) at 10M objects, 2^30 buckets 27% full,
 * 1410 + 227 us at 2M in dense spots, 2^28 buckets; the lists take 7.7 + 0.43
 * ms (6.5 TB/s of DRAM traffic, the copy's rate) and 1016 + 115 us.
 */
#include "glint_internal.cuh"

namespace glint {

constexpr int kIdThreads = 256;
constexpr int kIdWarps = kIdThreads / 32;
/* Records per lane in flight: with full lanes two are enough, and the registers
 * they save hold 40 warps per SM instead of 32 (four: 171 us at 1M objects, 2^26
 * buckets; two: 147; one: 145; two and spans of 512 or 2048: 148 and 192) */
constexpr int kIdIlp = 2;

/* Buckets per warp.  1024 amortises a block's start over many records; a
 * small table (below 2^23 buckets) would then be a handful of blocks, each
 * serially walking its span, so there a warp takes 128 (a 40k-bucket table:
 * 19 us at 1024, 5 blocks; 4.6 us at 128, 40 blocks). */
constexpr uint32_t kIdSpan = 1024, kIdSpanSmall = 128;
constexpr uint64_t kIdSmallBuckets = 1ull << 23;

uint32_t identify_span(uint64_t B) { return B < kIdSmallBuckets ? kIdSpanSmall : kIdSpan; }
uint64_t identify_tiles(uint64_t B) {
    const uint64_t tile = (uint64_t)identify_span(B) * kIdWarps;
    return (B + tile - 1) / tile;
}

/* the bytes of w equal to v, one bit each */
__device__ inline uint32_t byte_bits(uint32_t w, uint32_t v) {
    const uint32_t m = __vcmpeq4(w, v * 0x01010101u) & 0x08040201u; /* bits 0, 9, 18 and 27 */
    return (m | (m >> 8) | (m >> 16) | (m >> 24)) & 0xfu;
}
__device__ inline uint32_t emit_byte_bits(uint32_t w) { return byte_bits(w, kStampEmit); }

/* warp-collective: the span's stamps into shared memory */
template <uint32_t kSpan>
__device__ inline void load_stamps(const uint8_t *stamp, uint64_t wbase, uint8_t *sst) {
    const uint4 *src = reinterpret_cast<const uint4 *>(stamp + wbase);
    uint4 *dst = reinterpret_cast<uint4 *>(sst);
    for (uint32_t i = threadIdx.x & 31; i < kSpan / 16; i += 32) dst[i] = src[i];
    __syncwarp();
}

/* kStamps: an entry that the step touched has its stamp, else its tag */
template <uint32_t kSpan, bool kStamps>
__global__ void __launch_bounds__(kIdThreads) k_expire_count(uint8_t *__restrict__ stamp,
                                                             uint32_t *__restrict__ newline,
                                                             TRec *__restrict__ tab, uint64_t B, uint32_t min_plus1,
                                                             uint32_t *__restrict__ tile_cnt,
                                                             const float2 *__restrict__ fpos, uint32_t N,
                                                             DevCounters *cnt) {
    __shared__ uint32_t red[3][kIdWarps];
    __shared__ __align__(16) uint8_t sst[kIdWarps][kSpan];
    __shared__ uint16_t slist[kIdWarps][kSpan];
    __shared__ uint32_t snl[kIdWarps][kSpan / 128];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const uint64_t wbase = ((uint64_t)blockIdx.x * kIdWarps + wid) * kSpan;
    const uint32_t cur_time = cnt->step_time, st_now = cnt->step_tag;
    /* stamps and new-line words are allocated to a whole number of tiles */
    if (lane < (int)(kSpan / 128)) {
        /* the warp's lines filled this step; cleared for the next step */
        const uint32_t v = newline[(wbase >> 7) + lane];
        snl[wid][lane] = v;
        if (v) newline[(wbase >> 7) + lane] = 0;
    }
    load_stamps<kSpan>(stamp, wbase, sst[wid]);
    /* the span's buckets whose record is needed, 16 per lane at a time */
    uint32_t n = 0, kept = 0;
#pragma unroll
    for (uint32_t i0 = 0; i0 < kSpan; i0 += 512) {
        const uint32_t off = i0 + lane * 16;
        uint32_t bits = 0;
        if (off < kSpan && wbase + off < B) {
            const uint4 v = *reinterpret_cast<const uint4 *>(&sst[wid][off]);
            const uint32_t empty =
                byte_bits(v.x, 0) | (byte_bits(v.y, 0) << 4) | (byte_bits(v.z, 0) << 8) | (byte_bits(v.w, 0) << 12);
            bits = ~empty & 0xffffu;
            if (kStamps) {
                /* entries that stay need nothing of their records */
                const uint32_t now = kStampTouched + st_now;
                const uint32_t stay = byte_bits(v.x, now) | (byte_bits(v.y, now) << 4) | (byte_bits(v.z, now) << 8) |
                                      (byte_bits(v.w, now) << 12);
                kept += __popc(stay);
                bits &= ~stay;
            }
            /* every empty slot of a line that received a pair */
            const uint32_t lines = (snl[wid][off >> 7] >> ((off >> 2) & 31)) & 0xfu;
            bits |= ((lines & 1u) | ((lines & 2u) << 3) | ((lines & 4u) << 6) | ((lines & 8u) << 9)) * 0xfu & empty;
            const uint64_t left = B - (wbase + off);
            bits &= left < 16 ? (1u << left) - 1u : 0xffffu;
        }
        uint32_t incl = __popc(bits);
        const uint32_t mine = incl;
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += y;
        }
        uint32_t at = n + incl - mine;
        n += __shfl_sync(0xffffffffu, incl, 31);
        for (; bits; bits &= bits - 1) slist[wid][at++] = (uint16_t)(off + __ffs(bits) - 1);
    }
    __syncwarp();
    uint32_t emit = 0, taken = kept, active = kept;
    bool changed = false;
    for (uint32_t r0 = 0; r0 < n; r0 += 32 * kIdIlp) {
        uint32_t off[kIdIlp];
        bool fresh[kIdIlp];
        ulonglong2 rec[kIdIlp];
        float2 A[kIdIlp], Bp[kIdIlp];
#pragma unroll
        for (int u = 0; u < kIdIlp; ++u) {
            const uint32_t i = r0 + u * 32 + lane;
            off[u] = i < n ? slist[wid][i] : 0xffffffffu;
            rec[u] = make_ulonglong2(kEmptyW0, 0ull);
            if (off[u] != 0xffffffffu) rec[u] = *reinterpret_cast<const ulonglong2 *>(&tab[wbase + off[u]]);
        }
        /* a slot of a line that received a pair this step: empty, or the pair
         * (key word with kNewFlag).  Its start is now and its box that of its
         * two points (geometry.cu:481-489). */
#pragma unroll
        for (int u = 0; u < kIdIlp; ++u) {
            fresh[u] = off[u] != 0xffffffffu && sst[wid][off[u]] == kStampEmpty && rec[u].x != kEmptyW0 &&
                       (rec[u].x & kNewFlag);
            if (fresh[u]) {
                const uint32_t pa = pair_a(rec[u].x), pb = pair_b(rec[u].x);
                if (pa < N && pb < N) {
                    A[u] = fpos[pa];
                    Bp[u] = fpos[pb];
                }
            }
        }
#pragma unroll
        for (int u = 0; u < kIdIlp; ++u) {
            if (off[u] == 0xffffffffu) continue;
            TRec &r = tab[wbase + off[u]];
            if (fresh[u]) {
                ++taken;
                ++active;
                const unsigned long long pw = rec[u].x & kPairMask;
                TRec nr;
                nr.w0 = pw;
                nr.w1 = ((unsigned long long)st_now << 32) | cur_time;
                if (pair_a(pw) < N && pair_b(pw) < N) {
                    nr.mbr[0] = min(fenc(A[u].x), fenc(Bp[u].x));
                    nr.mbr[1] = min(fenc(A[u].y), fenc(Bp[u].y));
                    nr.mbr[2] = max(fenc(A[u].x), fenc(Bp[u].x));
                    nr.mbr[3] = max(fenc(A[u].y), fenc(Bp[u].y));
                } else {
                    atomicOr(&cnt->error_flags, GLINT_EF_DUPLICATE_NEW);
                    nr.mbr[0] = nr.mbr[1] = nr.mbr[2] = nr.mbr[3] = 0;
                }
                r = nr;
                sst[wid][off[u]] = kStamps ? (uint8_t)(kStampTouched + st_now) : (uint8_t)kStampOld;
                changed = true;
                continue;
            }
            if (sst[wid][off[u]] == kStampEmpty) continue;
            ++taken;
            const unsigned long long w1 = rec[u].y;
            if (!kStamps && (uint32_t)(w1 >> 32) == st_now) {
                ++active;
                continue;
            }
            changed = true;
            if (cur_time - (uint32_t)w1 >= min_plus1) {
                ++emit;
                sst[wid][off[u]] = kStampEmit;
            } else {
                *reinterpret_cast<ulonglong2 *>(&r) = make_ulonglong2(kEmptyW0, 0ull);
                sst[wid][off[u]] = kStampEmpty;
            }
        }
    }
    if (__any_sync(0xffffffffu, changed)) {
        uint4 *dst = reinterpret_cast<uint4 *>(stamp + wbase);
        const uint4 *src = reinterpret_cast<const uint4 *>(sst[wid]);
        for (uint32_t i = lane; i < kSpan / 16; i += 32) dst[i] = src[i];
    }
    emit = __reduce_add_sync(0xffffffffu, emit);
    taken = __reduce_add_sync(0xffffffffu, taken);
    active = __reduce_add_sync(0xffffffffu, active);
    if (lane == 0) {
        red[0][wid] = emit;
        red[1][wid] = taken;
        red[2][wid] = active;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t e = 0, t = 0, a = 0;
        for (int i = 0; i < kIdWarps; ++i) {
            e += red[0][i];
            t += red[1][i];
            a += red[2][i];
        }
        tile_cnt[blockIdx.x] = e;
        if (t) atomicAdd(&cnt->taken, (unsigned long long)t);
        if (a) atomicAdd(&cnt->active, a);
    }
}

/* Pass 2: the reports of tiles that have any, in bucket order, into the
 * meeting log.  A warp reads its stamps 16 at a time, lists the reports of
 * its span in order and writes them with consecutive lanes.  With few tiles
 * (kOwnScan) a block adds up the counts before its own itself, which costs
 * less than the scan's launch. */
template <uint32_t kSpan, bool kOwnScan>
__global__ void __launch_bounds__(kIdThreads) k_expire_emit(uint8_t *__restrict__ stamp, TRec *__restrict__ tab,
                                                            const uint32_t *__restrict__ tile_cnt,
                                                            uint32_t *__restrict__ tile_off,
                                                            glint_meeting *__restrict__ log, uint64_t log_cap,
                                                            const DevCounters *cnt) {
    __shared__ uint32_t ws[kIdWarps];
    __shared__ uint16_t slist[kIdWarps][kSpan];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    uint32_t before = 0;
    if (kOwnScan) {
        /* the last block also leaves the total */
        const bool last = blockIdx.x == gridDim.x - 1;
        if (tile_cnt[blockIdx.x] == 0 && !last) return; /* uniform per block */
        uint32_t v = 0;
        for (uint32_t i = threadIdx.x; i < blockIdx.x; i += kIdThreads) v += tile_cnt[i];
        v = __reduce_add_sync(0xffffffffu, v);
        if (lane == 0) ws[wid] = v;
        __syncthreads();
        for (int w = 0; w < kIdWarps; ++w) before += ws[w];
        __syncthreads();
        if (last && threadIdx.x == 0) tile_off[gridDim.x] = before + tile_cnt[blockIdx.x];
    } else {
        if (tile_cnt[blockIdx.x] == 0) return; /* uniform per block */
        before = tile_off[blockIdx.x];
    }
    const uint64_t wbase = ((uint64_t)blockIdx.x * kIdWarps + wid) * kSpan;
    uint4 *st = reinterpret_cast<uint4 *>(stamp + wbase);
    uint32_t n = 0;
#pragma unroll
    for (uint32_t i0 = 0; i0 < kSpan / 16; i0 += 32) {
        const uint32_t i = i0 + lane;
        uint4 v = make_uint4(0, 0, 0, 0);
        if (i < kSpan / 16) v = st[i];
        uint32_t bits = emit_byte_bits(v.x) | (emit_byte_bits(v.y) << 4) | (emit_byte_bits(v.z) << 8) | (emit_byte_bits(v.w) << 12);
        uint32_t incl = __popc(bits);
        const uint32_t mine = incl;
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += y;
        }
        uint32_t at = n + incl - mine;
        n += __shfl_sync(0xffffffffu, incl, 31);
        if (bits) {
            /* the reported entries leave: their stamps become empty */
            v.x &= ~__vcmpeq4(v.x, kStampEmit * 0x01010101u);
            v.y &= ~__vcmpeq4(v.y, kStampEmit * 0x01010101u);
            v.z &= ~__vcmpeq4(v.z, kStampEmit * 0x01010101u);
            v.w &= ~__vcmpeq4(v.w, kStampEmit * 0x01010101u);
            st[i] = v;
            for (; bits; bits &= bits - 1) slist[wid][at++] = (uint16_t)(i * 16 + __ffs(bits) - 1);
        }
    }
    if (lane == 0) ws[wid] = n;
    __syncthreads();
    uint64_t pos = cnt->log_head + before;
    for (int w = 0; w < wid; ++w) pos += ws[w];
    const uint32_t cur_time = cnt->step_time;
    for (uint32_t i = lane; i < n; i += 32) {
        TRec &r = tab[wbase + slist[wid][i]];
        const ulonglong2 k = *reinterpret_cast<const ulonglong2 *>(&r);
        const uint4 mb = *reinterpret_cast<const uint4 *>(r.mbr);
        uint4 *out = reinterpret_cast<uint4 *>(&log[(pos + i) % log_cap]);
        out[0] = make_uint4(pair_a(k.x), pair_b(k.x), (uint32_t)k.y, cur_time - 1);
        out[1] = make_uint4(__float_as_uint(fdec(mb.x)), __float_as_uint(fdec(mb.y)), __float_as_uint(fdec(mb.z)),
                            __float_as_uint(fdec(mb.w)));
        *reinterpret_cast<ulonglong2 *>(&r) = make_ulonglong2(kEmptyW0, 0ull);
    }
}

/* up to here a block's own sum is four loads per thread */
constexpr unsigned kOwnScanTiles = 1024;
uint32_t identify_launches(uint64_t tiles) { return tiles <= kOwnScanTiles ? 2u : 3u; }

template <uint32_t kSpan>
static void identify_passes(glint_ctx *c) {
    cudaStream_t s = c->stream;
    const unsigned tiles = (unsigned)c->n_tiles;
    const uint32_t min_plus1 = c->cfg.min_meet_time + 1;
    if (c->B <= kStampTouchBuckets)
        k_expire_count<kSpan, true><<<tiles, kIdThreads, 0, s>>>(c->d_stamp, c->d_newline, c->d_tab, c->B, min_plus1,
                                                                 c->d_tile_cnt, c->d_fpos, c->N, c->d_cnt);
    else
        k_expire_count<kSpan, false><<<tiles, kIdThreads, 0, s>>>(c->d_stamp, c->d_newline, c->d_tab, c->B, min_plus1,
                                                                  c->d_tile_cnt, c->d_fpos, c->N, c->d_cnt);
    if (tiles <= kOwnScanTiles) {
        k_expire_emit<kSpan, true><<<tiles, kIdThreads, 0, s>>>(c->d_stamp, c->d_tab, c->d_tile_cnt, c->d_tile_off,
                                                                c->d_log, c->log_cap, c->d_cnt);
        return;
    }
    scan_u32(c->d_tile_cnt, c->d_tile_off, tiles, c->d_scan_tmp, s);
    k_expire_emit<kSpan, false><<<tiles, kIdThreads, 0, s>>>(c->d_stamp, c->d_tab, c->d_tile_cnt, c->d_tile_off,
                                                             c->d_log, c->log_cap, c->d_cnt);
}

/* The step's reports are counted by tile_off[tiles]; the log's head moves in
 * the step's tail. */
cudaError_t launch_identify(glint_ctx *c, uint32_t cur_time) {
    (void)cur_time;
    if (identify_span(c->B) == kIdSpan) identify_passes<kIdSpan>(c);
    else identify_passes<kIdSpanSmall>(c);
    return cudaGetLastError();
}

} // namespace glint
