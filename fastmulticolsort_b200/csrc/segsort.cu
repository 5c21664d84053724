// segsort.cu -- (b) the per-round sort: a stable, segmented radix sort of
// (bank key, oid) pairs in HBM.
//
// Reference: Composer::sortByGroup<T> (src/composer.cpp:1222-1408) walks the
// previous round's groups and calls subsort -> Mergesort::avxmergesort_anytype
// (src/mergesort.h:2878-3096) once per group: block sorts with AVX2 bitonic
// networks, then 2-way merges, mallocing four buffers per group.  Round 0 is
// one group of n rows.
//
// B200 design.  Every group is a segment [start, start+len) that is sorted in
// place (segments never move).  Segments are binned by size:
//   len <= 16 (32)  one thread per segment, rows in registers;
//   len <= 256      one warp per segment, on chip;
//   len <= 8192     one CTA per segment, on chip;
//   larger          MSD radix levels: digit histograms per chunk of a segment,
//                   their prefixes, then a stable scatter without waits; every
//                   non-empty bucket becomes a child segment with 8 bits
//                   fewer, re-binned.
// The MSD scatter ranks keys by warp-level multi-split, so every pass is
// stable, and the on-chip sorts decide ties by position: the whole sort is
// stable, ties keep the oid order of the input, which is what the reference
// gives once its ties are canonicalised to ascending oid.  Rows move only
// through HBM in the levels; a smaller segment is read once and written once.
//
// Data sources of a segment: BUF0 (final buffer: the caller's order array and
// the sorted-key array), BUF1 (work buffer), EXT (the round's input: the bank
// gathered through the previous order, Composer::BATproject at
// src/composer.cpp:608-628, or the bank itself with iota oids in round 0).
#include "device_common.cuh"
#include "fmcs_internal.h"
#include "onchip.cuh"
#include "sort_lists.h"

#include <algorithm>
#include <functional>
#include <vector>

namespace fmcs {

namespace {

constexpr uint32_t kSrcBuf0 = 0;
constexpr uint32_t kSrcBuf1 = 1;
constexpr uint32_t kSrcExt = 2;
constexpr uint32_t kSkipBit = 0x100;

// Local tiers: a segment goes to the smallest tier whose capacity holds it, so
// that each kernel's unrolled item steps match the segment (few idle steps).
constexpr int kCapT = 16;    // thread per segment: registers, odd-even transposition network
constexpr int kCapT32 = 32;  // the same up to 32 rows, for 2- and 4-byte keys (own kernel: more registers)
constexpr int kItA = 4, kCapA = 32 * kItA;       // warp per segment: 128
constexpr int kItA2 = 8, kCapA2 = 32 * kItA2;    // 256
constexpr int kNtB1 = 64, kItB1 = 8, kCapB1 = kNtB1 * kItB1;    // CTA per segment: 512
constexpr int kNtB2 = 128, kItB2 = 8, kCapB2 = kNtB2 * kItB2;   // 1024
constexpr int kNtC1 = 256, kItC1 = 8, kCapC1 = kNtC1 * kItC1;   // 2048
constexpr int kNtC1b = 256, kItC1b = 9, kCapC1b = kNtC1b * kItC1b;   // 2304
constexpr int kNtC2 = 512, kItC2 = 8, kCapC2 = kNtC2 * kItC2;   // 4096
constexpr int kNtC3 = 1024, kItC3 = 8, kCapC3 = kNtC3 * kItC3;  // 8192
constexpr int kCapLocal = kCapC3;   // largest segment a local tier can take; larger: MSD levels
constexpr int kNtM = 256;           // MSD tile: 256 threads x IT items (IT = 8 or 16, tuned)
constexpr int kHistCtas = 4;         // resident histogram CTAs per SM (the grid is one wave)
constexpr int kMsdCtas16 = 3;       // resident scatter CTAs per SM with 16 rows per thread

// counters slot words
constexpr int kCtrMsdTile = 1;      // the scatter's next chunk
constexpr int kCtrLarge0 = 2;   // + level parity
constexpr int kCtrLocalA = 4;
constexpr int kCtrLocalA2 = 20;
constexpr int kCtrLocalB1 = 5;
constexpr int kCtrLocalB2 = 6;
constexpr int kCtrCopy = 7;
constexpr int kCtrMoved = 8;    // rows the current level's scatter moves
constexpr int kCtrLocalC1 = 9;
constexpr int kCtrLocalC2 = 10;
constexpr int kCtrLocalT = 11;
constexpr int kCtrLocalT32 = 14;
constexpr int kCtrCopyLarge = 12;   // copy entries larger than kCopySplit rows
constexpr int kCtrCopyTile = 13;
constexpr int kCtrLevel = 15;      // MSD levels started so far (device-side level index)
constexpr int kCtrLocalC3 = 16;
constexpr int kCtrLocalC1b = 17;
constexpr int kCtrWork = 18;       // chunks the current level's scatter moves
constexpr int kCtrLong = 19;       // super rows of the level's long segments (level_prefix_kernel)
constexpr int kCtrWords = kHostCounterWords;

// An HBM level cuts each large segment into chunks of a few tiles (chunk_rows
// rows, msd_chunk_rows).  A chunk has its own histogram row, counted by the CTA
// that reads it; msd_plan turns the rows of a segment into absolute digit bases
// (where the chunk's rows of a digit go), so the scatter's CTAs wait for
// nothing: a CTA takes a chunk and moves its tiles one after the other, its
// digit bases running on in registers.  Every kSuper chunks of a segment also
// share a super row, the sum of theirs, so that no plan CTA walks more than
// kSuper chunk rows and a few super rows.
// Chunk size: one tile as long as there are fewer than 32,768 (each is flushed
// and planned).  Larger chunks cost: the scatter's last round over its 444
// resident CTAs is as long as a chunk, and neighbouring tiles, whose rows share
// the ends of every digit's run, are then written far apart in time, so that
// half-filled lines leave L2 (16.8M rows: a level 108 us with one tile a
// chunk, 132 with two, 148 with five and 190 MB read instead of 134; a 67M-row
// Zipf plan 3.43 ms with one, 3.55 with two, 3.68 with four).
constexpr uint64_t kChunksWanted = 16384;
constexpr uint32_t kSuper = kTopSuper;

struct LargeSeg {
    uint32_t start, len, shift, src;
};

// A chunk to scatter: rows [start, start + len) of a segment, its histogram
// row, and the segment's remaining key bits and source (shift | src << 8).
struct Chunk {
    uint32_t start, len, row, info;
};

// The two alternating sets of an MSD level's buffers (large-segment list and
// the segments' digit totals; level L reads set L & 1 and fills set (L + 1) & 1).
// With dev_level the level index is read on the device (ctr[kCtrLevel]), so a
// level's launches are the same for every level (one graph body that loops);
// otherwise every launch works on set 0.
// (Kernels select a set with a conditional, not by indexing with the level
// parity: a parameter array indexed at run time is copied to local memory.)
struct LevelRefs {
    LargeSeg *large[2];
    uint32_t *super[2];       // kRadix words per super row (super_row)
    uint32_t *hist;           // kRadix words per chunk: its rows by digit, then its digit bases
    uint32_t *chunk_prefix;   // per large segment, its first chunk (level_prefix_kernel)
    uint2 *long_rows;         // (segment, super row of it) of the segments of more than kSuper chunks
    Chunk *work;              // the chunks to scatter (msd_plan)
    uint32_t *ctr;
    uint32_t chunk_rows, max_chunks;   // max_chunks: n / chunk_rows
    int dev_level;
    // level 0 (one segment) was counted before the sort, by the stitch: its
    // chunks' rows and after them their super rows
    const uint32_t *top_hist;
    // level 0's histogram pass leaves the keys it gathers through the order in
    // BUF0, beside the order itself: from then on the segments are BUF0's
    int gathered;
};

// The first super row of segment s, whose first chunk is c0.  (Rounding c0
// down and counting the segments before it leaves room for every segment's.)
__device__ __forceinline__ uint32_t super_row(uint32_t c0, uint32_t s) { return c0 / kSuper + s; }
// Super rows of a level of nseg segments, at most.
__host__ __device__ __forceinline__ uint64_t super_rows_max(uint64_t max_chunks, uint64_t nseg)
{
    return (max_chunks + nseg) / kSuper + nseg + 1;
}
__host__ __device__ __forceinline__ uint32_t seg_chunks(uint32_t len, uint32_t chunk_rows)
{
    return (len - 1) / chunk_rows + 1;   // len >= 1
}

// Index of the level whose launches are running (level_prefix_kernel has
// already advanced the counter for it).
__device__ __forceinline__ uint32_t running_level(const LevelRefs &r)
{
    return r.dev_level ? *(volatile const uint32_t *)&r.ctr[kCtrLevel] - 1u : 0u;
}

template <typename K>
struct Bufs {
    K *k0, *k1;
    uint32_t *v0, *v1;
    const K *ext_bank;
    const uint32_t *ext_order;   // NULL: iota
    // Per row, in the sorted order: 1 where its key differs from the row before
    // in its segment, or a segment starts (NULL: not wanted).  Whoever puts a
    // segment in its final order writes them, with the keys at hand: the group
    // ids then read a byte a row, and the sorted keys are not written.
    uint8_t *flags;
    int write_keys;   // 1 without flags
};

template <typename K>
__device__ __forceinline__ void load_kv(const Bufs<K> &b, uint32_t src, uint64_t i, K &k, uint32_t &v)
{
    if (src == kSrcExt) {
        if (b.ext_order) {
            v = b.ext_order[i];
            k = b.ext_bank[v];
        } else {
            v = (uint32_t)i;
            k = b.ext_bank[i];
        }
    } else if (src == kSrcBuf1) {
        k = b.k1[i];
        v = b.v1[i];
    } else {
        k = b.k0[i];
        v = b.v0[i];
    }
}

// A segment's rows into registers: warp-striped positions wbase + j*32 + lane
// (j < steps, position < len); the source switch is taken once per segment.
template <typename K, int IT>
__device__ __forceinline__ void load_rows(const Bufs<K> &b, uint32_t src, uint32_t start, uint32_t len, uint32_t steps,
                                          uint32_t wbase, K (&key)[IT], uint32_t (&val)[IT])
{
    const uint32_t lane = threadIdx.x & 31;
    if (src == kSrcExt && b.ext_order) {
        const uint32_t *os = b.ext_order + start;
#pragma unroll
        for (int j = 0; j < IT; ++j) {
            const uint32_t p = wbase + j * 32 + lane;
            val[j] = (j < (int)steps && p < len) ? os[p] : 0u;
        }
#pragma unroll
        for (int j = 0; j < IT; ++j) {
            const uint32_t p = wbase + j * 32 + lane;
            key[j] = (j < (int)steps && p < len) ? b.ext_bank[val[j]] : K(0);
        }
    } else if (src == kSrcExt) {
        const K *ks = b.ext_bank + start;
#pragma unroll
        for (int j = 0; j < IT; ++j) {
            const uint32_t p = wbase + j * 32 + lane;
            const bool ok = j < (int)steps && p < len;
            key[j] = ok ? ks[p] : K(0);
            val[j] = start + p;
        }
    } else {
        const K *ks = (src == kSrcBuf1 ? b.k1 : b.k0) + start;
        const uint32_t *vs = (src == kSrcBuf1 ? b.v1 : b.v0) + start;
#pragma unroll
        for (int j = 0; j < IT; ++j) {
            const uint32_t p = wbase + j * 32 + lane;
            const bool ok = j < (int)steps && p < len;
            key[j] = ok ? ks[p] : K(0);
            val[j] = ok ? vs[p] : 0u;
        }
    }
}

__device__ __forceinline__ uint2 pack_local(uint32_t start, uint32_t len, uint32_t shift, uint32_t src)
{
    return make_uint2(start, len | (shift << 16) | (src << 24));
}

struct Lists {
    uint2 *t, *t32, *a, *a2, *b1, *b2, *c1, *c1b, *c2, *c3;
    uint32_t cap_t32;      // kCapT32 for keys of <= 4 bytes, else 0 (17..32 rows go to the warp tier)
    LargeSeg *copy;        // segments that only need to reach BUF0, <= kCopySplit rows (warp each)
    LargeSeg *copy_large;  // the same, larger: copied by tiles across the grid
    uint32_t local_max;   // segments above this size take the MSD levels (tuned, <= kCapLocal)
    uint8_t *flags;       // Bufs::flags
};

// Route a segment (child or initial) to its tier.  Segments that need no
// sorting (one row, or no key bits left) only need to reach BUF0.
// A slot in the list whose counter is ctr[which]: the active lanes of a warp
// that go to the same list take their slots with one atomicAdd (children of
// one segment mostly share a tier, so the counters are hot addresses).
__device__ __forceinline__ uint32_t alloc_slot(uint32_t *ctr, int which)
{
    const uint32_t mask = __activemask();
    const uint32_t peers = __match_any_sync(mask, which);
    const int leader = __ffs(peers) - 1;
    uint32_t base = 0;
    if ((int)lane_id() == leader) base = atomicAdd(&ctr[which], (uint32_t)__popc(peers));
    base = __shfl_sync(mask, base, leader);
    return base + __popc(peers & lanemask_lt());
}

__device__ __forceinline__ int route_segment(uint32_t start, uint32_t len, uint32_t shift, uint32_t src,
                                             uint32_t *ctr, int large_ctr, LargeSeg *large_out, const Lists &L)
{
    if (len == 0) return -1;
    int which;
    if (len == 1 || shift == 0) {
        if (L.flags) L.flags[start] = 1;
        // already in place (with flags, the copy kernels still write its other rows')
        if (src == kSrcBuf0 && (len == 1 || !L.flags)) return -1;
        which = len > kCopySplit ? kCtrCopyLarge : kCtrCopy;
    } else if (len > L.local_max) {
        which = large_ctr;
    } else if (len <= (uint32_t)kCapT) {
        which = kCtrLocalT;
    } else if (len <= L.cap_t32) {
        which = kCtrLocalT32;
    } else if (len <= (uint32_t)kCapA) {
        which = kCtrLocalA;
    } else if (len <= (uint32_t)kCapA2) {
        which = kCtrLocalA2;
    } else if (len <= (uint32_t)kCapB1) {
        which = kCtrLocalB1;
    } else if (len <= (uint32_t)kCapB2) {
        which = kCtrLocalB2;
    } else if (len <= (uint32_t)kCapC1) {
        which = kCtrLocalC1;
    } else if (len <= (uint32_t)kCapC1b) {
        which = kCtrLocalC1b;
    } else if (len <= (uint32_t)kCapC2) {
        which = kCtrLocalC2;
    } else if (len <= (uint32_t)kCapC3) {
        which = kCtrLocalC3;
    } else {
        which = large_ctr;
    }
    const uint32_t slot = alloc_slot(ctr, which);
    const uint2 e = pack_local(start, len, shift, src);
    switch (which) {
    case kCtrCopyLarge: L.copy_large[slot] = LargeSeg{start, len, 0, src}; break;
    case kCtrCopy: L.copy[slot] = LargeSeg{start, len, 0, src}; break;
    case kCtrLocalT: L.t[slot] = e; break;
    case kCtrLocalT32: L.t32[slot] = e; break;
    case kCtrLocalA: L.a[slot] = e; break;
    case kCtrLocalA2: L.a2[slot] = e; break;
    case kCtrLocalB1: L.b1[slot] = e; break;
    case kCtrLocalB2: L.b2[slot] = e; break;
    case kCtrLocalC1: L.c1[slot] = e; break;
    case kCtrLocalC1b: L.c1b[slot] = e; break;
    case kCtrLocalC2: L.c2[slot] = e; break;
    case kCtrLocalC3: L.c3[slot] = e; break;
    default: large_out[slot] = LargeSeg{start, len, shift, src};
    }
    return which;
}

// ---------------------------------------------------------------------------
// classification of the round's initial segments
// ---------------------------------------------------------------------------
template <typename K>
__global__ void classify_kernel(Bufs<K> b, const uint32_t *__restrict__ seg_start, const uint32_t *d_nseg,
                                uint64_t n, uint32_t key_bits, uint32_t *ctr, LargeSeg *large0, Lists lists,
                                const uint32_t *top_hist, const uint32_t *d_key_bits,
                                const uint32_t *d_in_order, bool skip_single, bool mark_starts)
{
    kernel_prologue();
    if (d_key_bits) key_bits = min(key_bits, *d_key_bits);
    if (d_in_order && *d_in_order) {
        // Every segment is in order: the rows keep their places, and their keys and
        // oids go to BUF0 here.  (No segment is listed: there may be one per two
        // rows, many more than the levels' finished segments, which the copy lists
        // are sized for.)
        for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
            K k;
            uint32_t v;
            load_kv(b, kSrcExt, i, k, v);
            b.k0[i] = k;
            b.v0[i] = v;
        }
        return;
    }
    if (!seg_start && top_hist && n > lists.local_max) {
        // round 0 over the whole array with its first-level histogram already
        // counted (level 0's msd_plan reads the stitch's rows): the one large
        // segment
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            ctr[kCtrLarge0] = 1;
            large0[0] = LargeSeg{0, (uint32_t)n, key_bits, kSrcExt};
        }
        return;
    }
    if (!seg_start) {
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            if (n == 1) {
                K k;
                uint32_t v;
                load_kv(b, kSrcExt, 0, k, v);
                b.k0[0] = k;
                b.v0[0] = v;
                if (b.flags) b.flags[0] = 1;
            } else {
                route_segment(0u, (uint32_t)n, key_bits, kSrcExt, ctr, kCtrLarge0, large0, lists);
            }
        }
        return;
    }
    // 128 segments a warp.  First four a lane, their starts in one 16-byte load
    // (seg_start is 16-byte aligned): where all are one row and nobody reads their
    // keys (a round after nearly unique keys) the kernel only streams the starts.
    // 67M of them: 126 us one segment a thread, 57 so.  Otherwise the warp takes
    // them 32 at a time, a lane each, so that neighbours stay neighbours in their
    // list, as the tiers read it (four a lane made rounds of 2 to 16 rows a segment
    // 4 to 8% slower).
    const uint32_t nseg = *d_nseg;
    const uint32_t lane = lane_id();
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x * 4;
    for (uint64_t w0 = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x - lane) * 4; w0 < nseg; w0 += stride) {
        const uint64_t s0 = w0 + lane * 4;
        bool ones = skip_single && s0 + 4 <= nseg;
        uint32_t first = 0;
        if (ones) {
            const uint4 w = *reinterpret_cast<const uint4 *>(seg_start + s0);
            first = w.x;
            // (starts increase but for empty segments)
            ones = w.y - w.x == 1 && w.z - w.y == 1 && w.w - w.z == 1 && seg_start[s0 + 4] - w.w == 1;
        }
        if (__all_sync(0xFFFFFFFFu, ones)) {
            if (mark_starts) {
#pragma unroll
                for (uint32_t k = 0; k < 4; ++k) b.flags[first + k] = 1;
            }
            continue;
        }
#pragma unroll 1
        for (uint32_t k = 0; k < 4; ++k) {
            const uint64_t s = w0 + k * 32 + lane;
            if (s >= nseg) break;
            const uint32_t start = seg_start[s], len = seg_start[s + 1] - start;
            if (mark_starts && len) b.flags[start] = 1;
            if (len == 1) {
                // A one-row segment keeps its position.  With skip_single its
                // oid is in BUF0 already and nothing reads its key: nothing to
                // do.  (Fetching those keys was a random 32-byte sector per
                // row: 1.25 ms of the second round of a 67M-row plan whose
                // first round leaves one-row groups.)
                if (skip_single) continue;
                // Otherwise copy it straight to BUF0.
                K key;
                uint32_t v;
                load_kv(b, kSrcExt, start, key, v);
                if (b.write_keys) b.k0[start] = key;
                b.v0[start] = v;
                continue;
            }
            route_segment(start, len, key_bits, kSrcExt, ctr, kCtrLarge0, large0, lists);
        }
    }
}

// ---------------------------------------------------------------------------
// MSD level kernels (large segments)
// ---------------------------------------------------------------------------
// Exclusive prefix of the tile (or chunk) counts of the listed segments (one CTA).
// With long_rows, the super rows of the segments of more than kSuper tiles are
// listed there (*nlong of them).
__device__ __forceinline__ void tile_prefix_body(const LargeSeg *segs, uint32_t nseg, uint32_t *tile_prefix,
                                                 uint32_t tile_rows, uint2 *long_rows = nullptr,
                                                 uint32_t *nlong = nullptr)
{
    __shared__ uint32_t warp_sums[32];
    __shared__ uint32_t carry;
    if (threadIdx.x == 0) carry = 0;
    __syncthreads();
    for (uint32_t base = 0; base < nseg; base += blockDim.x) {
        const uint32_t s = base + threadIdx.x;
        const uint32_t c = s >= nseg ? 0u : seg_chunks(segs[s].len, tile_rows);
        if (long_rows && c > kSuper) {
            const uint32_t k = (c - 1) / kSuper + 1, at = atomicAdd(nlong, k);
            for (uint32_t i = 0; i < k; ++i) long_rows[at + i] = make_uint2(s, i);
        }
        uint32_t incl = c;
        for (int o = 1; o < 32; o <<= 1) {
            uint32_t y = __shfl_up_sync(0xFFFFFFFFu, incl, o);
            if ((int)lane_id() >= o) incl += y;
        }
        if (lane_id() == 31) warp_sums[threadIdx.x >> 5] = incl;
        __syncthreads();
        if (threadIdx.x < 32) {
            uint32_t v = threadIdx.x < blockDim.x / 32 ? warp_sums[threadIdx.x] : 0u;
            uint32_t vi = v;
            for (int o = 1; o < 32; o <<= 1) {
                uint32_t y = __shfl_up_sync(0xFFFFFFFFu, vi, o);
                if ((int)threadIdx.x >= o) vi += y;
            }
            warp_sums[threadIdx.x] = vi - v;
        }
        __syncthreads();
        const uint32_t excl = carry + warp_sums[threadIdx.x >> 5] + incl - c;
        if (s < nseg) tile_prefix[s] = excl;
        __syncthreads();
        if (threadIdx.x == blockDim.x - 1) carry = excl + c;
        __syncthreads();
    }
    if (threadIdx.x == 0) tile_prefix[nseg] = carry;
}

__global__ void __launch_bounds__(1024) tile_prefix_kernel(const LargeSeg *segs, const uint32_t *d_nseg,
                                                           uint32_t *tile_prefix, uint32_t *reset, uint32_t tile_rows)
{
    kernel_prologue();
    if (threadIdx.x == 0) *reset = 0;
    tile_prefix_body(segs, *d_nseg, tile_prefix, tile_rows);
}

// First launch of an MSD level: chunk prefix of the level's large segments,
// resets of the level's counters, and (device-side levels) the level index
// advanced for the level's other launches.
__global__ void __launch_bounds__(1024) level_prefix_kernel(LevelRefs r)
{
    kernel_prologue();
    const uint32_t lvl = r.dev_level ? r.ctr[kCtrLevel] : 0u;
    const uint32_t cur = lvl & 1u, nxt = cur ^ 1u;
    const uint32_t nseg = r.ctr[kCtrLarge0 + cur];
    __syncthreads();   // every thread has read the level index before it advances
    if (threadIdx.x == 0) {
        r.ctr[kCtrLarge0 + nxt] = 0;
        r.ctr[kCtrMsdTile] = 0;
        r.ctr[kCtrMoved] = 0;
        r.ctr[kCtrWork] = 0;
        r.ctr[kCtrLong] = 0;
        if (r.dev_level) r.ctr[kCtrLevel] = lvl + 1;
    }
    __syncthreads();
    tile_prefix_body(cur ? r.large[1] : r.large[0], nseg, r.chunk_prefix, r.chunk_rows, r.long_rows,
                     &r.ctr[kCtrLong]);
    if (lvl == 0 && !r.top_hist) {
        // level 0's super rows start at zero (a level's scatter zeroes the next level's)
        __syncthreads();
        const uint64_t words = nseg ? (uint64_t)(super_row(r.chunk_prefix[nseg], nseg) + 1) * (kRadix / 4) : 0;
        uint4 *h = reinterpret_cast<uint4 *>(r.super[0]);
        for (uint64_t i = threadIdx.x; i < words; i += blockDim.x) h[i] = make_uint4(0, 0, 0, 0);
    }
}

// Top-digit histogram of every chunk, added to its super row as well.  A CTA
// takes a contiguous run of chunks and reads whole ones, so a chunk's row is
// stored, not added to.  Each thread issues all of a tile's loads before
// counting (up to 16 in flight), and each warp counts into its own shared
// sub-histogram so that skewed digits do not serialize the whole block on one
// counter.  Two sets of them alternate by chunk: one is written out while the
// next chunk's loads are in flight, one barrier a chunk.
template <typename K>
__global__ void __launch_bounds__(kNtM, kHistCtas) msd_hist_kernel(Bufs<K> b, LevelRefs r)
{
    kernel_prologue();
    constexpr int NW = kNtM / 32;
    constexpr int MAXJ = 16;
    __shared__ uint32_t sh[2][NW][kRadix];
    const uint32_t lvl = running_level(r);
    if (lvl == 0 && r.top_hist) return;
    const uint32_t cur = lvl & 1u;
    const LargeSeg *segs = (cur ? r.large[1] : r.large[0]);
    uint32_t *super = (cur ? r.super[1] : r.super[0]);
    const uint32_t nseg = r.ctr[kCtrLarge0 + cur];
    if (nseg == 0) return;
    const uint32_t C = r.chunk_prefix[nseg];
    const uint32_t warp = threadIdx.x >> 5;
    const uint32_t per = (C + gridDim.x - 1) / gridDim.x;
    const uint32_t q0 = blockIdx.x * per, q1 = min(C, q0 + per);
    if (q0 >= C) return;
    for (int d = threadIdx.x; d < 2 * NW * kRadix; d += blockDim.x) (&sh[0][0][0])[d] = 0;
    uint32_t s = find_segment_warp(r.chunk_prefix, nseg, q0);
    LargeSeg sg = segs[s];
    uint32_t sfirst = r.chunk_prefix[s], snext = r.chunk_prefix[s + 1];
    uint32_t prow = 0, psup = 0;   // the chunk to write out
    // up to MAXJ rows a thread of the `rows` rows of the segment from row `beg`;
    // the source switch is taken once a tile
    auto load_tile = [&](K (&key)[MAXJ], uint32_t beg, uint32_t rows) {
        const uint64_t at = (uint64_t)sg.start + beg;
        if (sg.src == kSrcExt && b.ext_order) {
            const uint32_t *os = b.ext_order + at;
            uint32_t v[MAXJ];
#pragma unroll
            for (int j = 0; j < MAXJ; ++j) {
                const uint32_t i = threadIdx.x + j * kNtM;
                v[j] = i < rows ? os[i] : 0u;
            }
#pragma unroll
            for (int j = 0; j < MAXJ; ++j) {
                const uint32_t i = threadIdx.x + j * kNtM;
                key[j] = i < rows ? b.ext_bank[v[j]] : K(0);
            }
            if (r.gathered) {
                // the scatter reads them in order instead of gathering again
                // (32 bytes fetched a row): 60M rows in 64 groups, two rounds,
                // 3.23 -> 2.54 ms
                K *kd = b.k0 + at;
#pragma unroll
                for (int j = 0; j < MAXJ; ++j) {
                    const uint32_t i = threadIdx.x + j * kNtM;
                    if (i < rows) kd[i] = key[j];
                }
            }
        } else {
            const K *ks = (sg.src == kSrcExt ? b.ext_bank : sg.src == kSrcBuf1 ? b.k1 : b.k0) + at;
#pragma unroll
            for (int j = 0; j < MAXJ; ++j) {
                const uint32_t i = threadIdx.x + j * kNtM;
                key[j] = i < rows ? ks[i] : K(0);
            }
        }
    };
    __syncthreads();
    for (uint32_t q = q0; q <= q1; ++q) {
        const uint32_t set = (q - q0) & 1u;
        K key[MAXJ];
        uint32_t beg = 0, rows = 0, lo = 0, width = 0;   // (rows left: a row's index may end at 2^32 - 1)
        if (q < q1) {
            if (q >= snext) {   // every large segment has a chunk: the next chunk starts the next segment
                ++s;
                sg = segs[s];
                sfirst = snext;
                snext = r.chunk_prefix[s + 1];
            }
            width = sg.shift < (uint32_t)kRadixBits ? sg.shift : (uint32_t)kRadixBits;
            lo = sg.shift - width;
            beg = (q - sfirst) * r.chunk_rows;
            rows = min(r.chunk_rows, sg.len - beg);
            load_tile(key, beg, rows);
        }
        if (q > q0) {
            // the chunk before, counted in the other set
            const uint32_t d = threadIdx.x;
            uint32_t c = 0;
#pragma unroll
            for (int w = 0; w < NW; ++w) {
                c += sh[set ^ 1u][w][d];
                sh[set ^ 1u][w][d] = 0;
            }
            r.hist[(uint64_t)prow * kRadix + d] = c;
            if (c) atomicAdd(&super[(uint64_t)psup * kRadix + d], c);
        }
        if (q == q1) break;
        for (;;) {
#pragma unroll
            for (int j = 0; j < MAXJ; ++j) {
                const uint32_t i = threadIdx.x + j * kNtM;
                if (i < rows) atomicAdd(&sh[set][warp][digit_of(key[j], lo, width)], 1u);
            }
            if (rows <= MAXJ * kNtM) break;
            rows -= MAXJ * kNtM;
            beg += MAXJ * kNtM;
            load_tile(key, beg, rows);
        }
        prow = q;
        psup = super_row(sfirst, s) + (q - sfirst) / kSuper;
        __syncthreads();
    }
}

// Per large segment: its digit totals (the sum of its super rows), exclusive
// digit offsets, skip detection, children, its chunks' digit bases (the
// segment's start and offset of the digit plus the digit's rows in the earlier
// chunks), and its chunks listed for the scatter.  A segment of up to kSuper
// chunks is one CTA's work; of a longer one (a round's first level; skew) a CTA
// does each super row's chunks.  A thread per digit, kPlanLoads loads in flight.
constexpr int kPlanThreads = 256;
constexpr int kPlanLoads = 16;
static_assert(kPlanThreads == kRadix, "a thread per digit");

__global__ void __launch_bounds__(kPlanThreads) msd_plan_kernel(LevelRefs r, Lists lists, bool emit_children = true)
{
    kernel_prologue();
    __shared__ uint32_t cnt[kRadix];
    __shared__ uint32_t tmp[kPlanThreads / 32 + 1];
    __shared__ uint32_t s_skip, s_work;
    const uint32_t lvl = running_level(r);
    const uint32_t cur = lvl & 1u, nxt = cur ^ 1u;
    LargeSeg *segs = (cur ? r.large[1] : r.large[0]);
    LargeSeg *large_next = (nxt ? r.large[1] : r.large[0]);
    const uint32_t nseg = r.ctr[kCtrLarge0 + cur];
    if (nseg == 0) return;
    const bool top = lvl == 0 && r.top_hist;   // one segment, counted by the stitch
    const uint32_t *counts = top ? r.top_hist : r.hist;
    const uint32_t *super = top ? r.top_hist + (uint64_t)r.chunk_prefix[1] * kRadix
                                : (cur ? r.super[1] : r.super[0]);
    const uint32_t d = threadIdx.x;
    // Sum of digit d over rows [q, q1) of an array of rows.
    auto sum_rows = [&](const uint32_t *rows, uint32_t q, uint32_t q1) -> uint32_t {
        uint32_t c = 0;
        for (; q < q1; q += kPlanLoads) {
            uint32_t v[kPlanLoads];
#pragma unroll
            for (int j = 0; j < kPlanLoads; ++j) v[j] = q + j < q1 ? rows[(uint64_t)(q + j) * kRadix + d] : 0u;
#pragma unroll
            for (int j = 0; j < kPlanLoads; ++j) c += v[j];
        }
        return c;
    };
    // Exclusive digit offsets into cnt from the digit totals; true when one
    // digit holds every row (the pass is the identity).
    auto offsets = [&](uint32_t t, uint32_t len) -> bool {
        if (d == 0) s_skip = 0;
        __syncthreads();
        cnt[d] = t;
        if (t == len) s_skip = 1;
        uint32_t total;
        block_exclusive_scan_radix<kPlanThreads>(cnt, tmp, &total);
        return s_skip != 0;
    };
    // Chunk rows [q, q1) become bases, running on from `run`.
    auto write_bases = [&](uint32_t q, uint32_t q1, uint32_t run) {
        for (; q < q1; q += kPlanLoads) {
            uint32_t v[kPlanLoads];
#pragma unroll
            for (int j = 0; j < kPlanLoads; ++j) v[j] = q + j < q1 ? counts[(uint64_t)(q + j) * kRadix + d] : 0u;
#pragma unroll
            for (int j = 0; j < kPlanLoads; ++j) {
                if (q + j < q1) r.hist[(uint64_t)(q + j) * kRadix + d] = run;
                run += v[j];
            }
        }
    };
    const uint32_t nitems = r.ctr[kCtrLong];
    for (uint32_t i = gridDim.x - 1 - blockIdx.x; i < nitems; i += gridDim.x) {
        const uint2 it = r.long_rows[i];
        const LargeSeg sg = segs[it.x];
        const uint32_t r0 = r.chunk_prefix[it.x], r1 = r.chunk_prefix[it.x + 1];
        const uint32_t s0 = top ? 0u : super_row(r0, it.x), ns = (r1 - r0 - 1) / kSuper + 1;
        const uint32_t before = sum_rows(super, s0, s0 + it.y);
        const bool skip = offsets(before + sum_rows(super, s0 + it.y, s0 + ns), sg.len);
        const uint32_t q = r0 + it.y * kSuper;
        if (!skip) write_bases(q, min(r1, q + kSuper), sg.start + cnt[d] + before);
        __syncthreads();
    }
    for (uint32_t s = blockIdx.x; s < nseg; s += gridDim.x) {
        LargeSeg sg = segs[s];
        if (lvl == 0 && r.gathered) sg.src = kSrcBuf0;
        const uint32_t r0 = r.chunk_prefix[s], r1 = r.chunk_prefix[s + 1];
        const uint32_t s0 = top ? 0u : super_row(r0, s);
        const uint32_t tot = sum_rows(super, s0, s0 + (r1 - r0 - 1) / kSuper + 1);
        const bool skip = offsets(tot, sg.len);
        const uint32_t off = cnt[d];
        if (d == 0) {
            if (skip) {
                segs[s].src = sg.src | kSkipBit;
            } else {
                s_work = atomicAdd(&r.ctr[kCtrWork], r1 - r0);
                atomicAdd(&r.ctr[kCtrMoved], sg.len);
            }
        }
        if (!skip && r1 - r0 <= kSuper) write_bases(r0, r1, sg.start + off);
        __syncthreads();
        if (!skip) {
            for (uint32_t q = r0 + d; q < r1; q += kPlanThreads) {
                const uint32_t o = (q - r0) * r.chunk_rows;
                r.work[s_work + (q - r0)] = Chunk{sg.start + o, min(r.chunk_rows, sg.len - o), q,
                                                  sg.shift | (sg.src << 8)};
            }
        }
        if (emit_children && tot > 0) {
            const uint32_t width = sg.shift < (uint32_t)kRadixBits ? sg.shift : (uint32_t)kRadixBits;
            const uint32_t child_src = skip ? sg.src : (sg.src == kSrcBuf1 ? kSrcBuf0 : kSrcBuf1);
            route_segment(sg.start + off, tot, sg.shift - width, child_src, r.ctr, kCtrLarge0 + (int)nxt, large_next,
                          lists);
        }
        __syncthreads();
    }
}

// Resident CTAs of the scatter per SM (the launch bound and the grid).
constexpr int msd_ctas_per_sm(int it) { return it >= 16 ? kMsdCtas16 : 4; }

template <typename K, int IT>
struct MsdSmem {
    uint32_t whist[kNtM / 32][kRadix];   // per warp and digit: rows so far, then where they go in the tile
    uint32_t doff[kRadix];       // tile-local exclusive digit offsets
    uint32_t gdst[kRadix];       // global destination base per digit (mod 2^32; rows < 2^32)
    Chunk next;
    uint32_t tmp[kNtM / 32 + 4];
    K keys[kNtM * IT];
    uint32_t vals[kNtM * IT];
    static_assert(kNtM * IT >= (kNtM / 32) * kRadix, "the peer words of kRankOr fit in vals");
    static_assert(kNtM == kRadix, "a thread per digit");
};

// Moves the level's chunks: a CTA claims a chunk and takes its tiles in order.
// Per tile: rank (stable, by warp-level multi-split), digit offsets, rows staged
// in digit order, written out in runs.  As soon as a tile is staged its
// registers take the loads of the next one (of this chunk, or of the next
// chunk, claimed while this one's first tile was ranked), which so run during
// the write-out.
// Bound: the shared-memory pipe (83% busy; about 50 wavefronts per 32 rows: the
// peer word's OR, load and clear, the counter's load and store, the rank's
// base, staging both arrays and reading them back).  One level over 16.8M rows
// of 8-byte keys: 108 us, 24 bytes a row at 3.7 TB/s; 130 us when every tile
// also waited for its predecessors' digit counts (decoupled look-back).
// Counters and peer bits in one 64-bit word (fewer accesses, but 64-bit ones):
// 131 us; ballots instead of the OR: 117; match.any: 156.
template <typename K, int RANK, int IT>
__global__ void __launch_bounds__(kNtM, msd_ctas_per_sm(IT)) msd_scatter_kernel(Bufs<K> b, LevelRefs r,
                                                                                cudaGraphConditionalHandle more,
                                                                                uint32_t levels, uint32_t *host,
                                                                                uint32_t seq)
{
    kernel_prologue();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    MsdSmem<K, IT> &sm = *reinterpret_cast<MsdSmem<K, IT> *>(smem_raw);
    constexpr uint32_t kTileM = kNtM * IT;
    const uint32_t lvl = running_level(r);
    const uint32_t cur = lvl & 1u;
    // An eager call reads the counters back (the next level's count, the rows
    // moved, the tiers' list sizes, final since msd_plan) while this kernel runs.
    if (host && blockIdx.x == 0 && threadIdx.x < 32) publish_counters(r.ctr, host, seq);
    // Inside a graph, the level loop goes on while the next level has large
    // segments (msd_plan has counted them before this launch).
    const uint32_t nnext = r.ctr[kCtrLarge0 + (cur ^ 1u)];
    if (more && blockIdx.x == 0 && threadIdx.x == 0)
        cudaGraphSetConditional(more, (nnext > 0 && lvl + 1 < levels) ? 1u : 0u);
    {
        // the next level's super rows start at zero (they held the previous
        // level's, which nothing reads any more)
        uint4 *h = reinterpret_cast<uint4 *>(cur ? r.super[0] : r.super[1]);
        const uint64_t words = nnext ? super_rows_max(r.max_chunks, nnext) * (kRadix / 4) : 0;
        for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < words;
             i += (uint64_t)gridDim.x * blockDim.x)
            h[i] = make_uint4(0, 0, 0, 0);
    }
    const uint32_t C = r.ctr[kCtrWork];
    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const uint32_t wbase = warp * (IT * 32);
    // chunk number c of the list, or an empty one past its end
    auto chunk_at = [&](uint32_t c) -> Chunk { return c < C ? r.work[c] : Chunk{0, 0, 0, 0}; };
    if (threadIdx.x == 0) sm.next = chunk_at(atomicAdd(&r.ctr[kCtrMsdTile], 1u));
    __syncthreads();
    Chunk ck = sm.next;
    K key[IT];
    uint32_t val[IT];
    uint32_t gbase = 0;   // this thread's digit: where the chunk's next row of it goes
    if (ck.len) {
        load_rows<K, IT>(b, ck.info >> 8, ck.start, min(ck.len, kTileM), IT, wbase, key, val);
        gbase = r.hist[(uint64_t)ck.row * kRadix + threadIdx.x];
    }
    bool first = true;   // the chunk's first tile
    while (ck.len) {
        const uint32_t src = ck.info >> 8, shift = ck.info & 0xFFu;
        const uint32_t cnt = min(ck.len, kTileM);
        const uint32_t width = shift < (uint32_t)kRadixBits ? shift : (uint32_t)kRadixBits;
        const uint32_t lo = shift - width;
        uint32_t claimed = 0;
        if (first && threadIdx.x == 0) claimed = atomicAdd(&r.ctr[kCtrMsdTile], 1u);
        // kRankOr's per-warp peer words live in the vals staging area, which
        // is free until the ranks are known
        uint32_t *peerw = &sm.vals[warp * kRadix];
#pragma unroll
        for (int d = lane; d < kRadix / 4; d += 32) {
            reinterpret_cast<uint4 *>(sm.whist[warp])[d] = make_uint4(0, 0, 0, 0);
            if constexpr (RANK == kRankOr) reinterpret_cast<uint4 *>(peerw)[d] = make_uint4(0, 0, 0, 0);
        }
        __syncwarp();
        uint32_t rd[IT];   // rank in the warp (low 16 bits) | digit << 16
        if (cnt == kTileM && width == (uint32_t)kRadixBits) {
            // a whole tile and a whole digit (the common case): no lane checks
#pragma unroll
            for (int j = 0; j < IT; ++j) {
                const uint32_t d = (uint32_t)((uint64_t)key[j] >> lo) & (uint32_t)(kRadix - 1);
                if constexpr (RANK == kRankOr)
                    rd[j] = wlms_rank_or(d, true, sm.whist[warp], peerw) | (d << 16);
                else
                    rd[j] = wlms_rank_full<RANK>(d, sm.whist[warp]) | (d << 16);
            }
        } else {
#pragma unroll
            for (int j = 0; j < IT; ++j) {
                const uint32_t p = wbase + j * 32 + lane;
                const uint32_t d = digit_of(key[j], lo, width);
                if constexpr (RANK == kRankOr)
                    rd[j] = wlms_rank_or(d, p < cnt, sm.whist[warp], peerw) | (d << 16);
                else
                    rd[j] = wlms_rank<RANK>(d, p < cnt, sm.whist[warp], width) | (d << 16);
            }
        }
        if (first && threadIdx.x == 0) sm.next = chunk_at(claimed);
        __syncthreads();
        // this thread's digit: its rows per warp, tile total
        uint32_t wc[kNtM / 32], total = 0;
#pragma unroll
        for (int w = 0; w < kNtM / 32; ++w) {
            wc[w] = sm.whist[w][threadIdx.x];
            total += wc[w];
        }
        sm.doff[threadIdx.x] = total;
        __syncthreads();
        uint32_t tot;
        block_exclusive_scan_radix<kNtM>(sm.doff, sm.tmp, &tot);
        {
            uint32_t dof = sm.doff[threadIdx.x];
            sm.gdst[threadIdx.x] = gbase - dof;   // wraps; + slot is in range
            gbase += total;
#pragma unroll
            for (int w = 0; w < kNtM / 32; ++w) {
                sm.whist[w][threadIdx.x] = dof;
                dof += wc[w];
            }
        }
        __syncthreads();
#pragma unroll
        for (int j = 0; j < IT; ++j) {
            const uint32_t p = wbase + j * 32 + lane;
            if (p < cnt) {
                const uint32_t pos = sm.whist[warp][rd[j] >> 16] + (rd[j] & 0xFFFFu);
                sm.keys[pos] = key[j];
                sm.vals[pos] = val[j];
            }
        }
        __syncthreads();
        // the next tile's loads: the chunk's, or the first of the next chunk
        ck.start += cnt;
        ck.len -= cnt;
        first = ck.len == 0;
        if (first) {
            ck = sm.next;
            if (ck.len) gbase = r.hist[(uint64_t)ck.row * kRadix + threadIdx.x];
        }
        if (ck.len) load_rows<K, IT>(b, ck.info >> 8, ck.start, min(ck.len, kTileM), IT, wbase, key, val);
        K *dk = (src == kSrcBuf1) ? b.k0 : b.k1;
        uint32_t *dv = (src == kSrcBuf1) ? b.v0 : b.v1;
        for (uint32_t i = threadIdx.x; i < cnt; i += kNtM) {
            const K kk = sm.keys[i];
            const uint32_t o = sm.gdst[digit_of(kk, lo, width)] + i;
            dk[o] = kk;
            dv[o] = sm.vals[i];
        }
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------
// local tiers
// ---------------------------------------------------------------------------
// One segment, on chip (onchip.cuh): one HBM read and one write per row.
// FLAGS: it writes the rows' flags, otherwise their keys.
template <typename K, int NT, int IT, bool FLAGS>
__device__ __forceinline__ void onchip_sort(OnchipSmem<K, NT, IT> &sm, const Bufs<K> &b, uint32_t start, uint32_t len,
                                            uint32_t src)
{
    const uint32_t lane = lane_id();
    const uint32_t tid = NT == 32 ? lane : threadIdx.x;
    // The rows are spread evenly over the warps: warp w holds positions
    // [w*steps*32, (w+1)*steps*32), a step is one row per lane.
    const uint32_t steps = (len + NT - 1) / NT;
    const uint32_t wbase = (NT == 32 ? 0u : threadIdx.x >> 5) * steps * 32;
    unsigned long long c[IT];
    {
        K key[IT];
        uint32_t val[IT];
        load_rows<K, IT>(b, src, start, len, steps, wbase, key, val);
#pragma unroll
        for (int j = 0; j < IT; ++j) {
            const uint32_t p = wbase + j * 32 + lane;
            c[j] = (unsigned long long)key[j];
            if (j < (int)steps && p < len) sm.vals[p] = val[j];
        }
    }
    const OnchipInfo f = onchip_core<K, NT, IT>(sm, c, steps, wbase, len);
    K *ko = b.k0 + start;
    uint32_t *vo = b.v0 + start;
    uint8_t *fo = b.flags + start;
    if (f.same) {
#pragma unroll
        for (int j = 0; j < IT; ++j) {
            const uint32_t p = wbase + j * 32 + lane;
            if (j < (int)steps && p < len) {
                if (src != kSrcBuf0) {
                    if (!FLAGS) ko[p] = (K)c[j];
                    vo[p] = sm.vals[p];
                }
                if (FLAGS) fo[p] = p == 0;
            }
        }
    } else {
        // every load of this segment is done (the sort's barriers) before the
        // first store into BUF0, which may alias the EXT oids of the range
        const uint32_t pmask = (1u << f.nbits) - 1u;
        for (uint32_t p = tid; p < len; p += NT) {
            const unsigned long long x = sm.cs[p];
            const uint32_t q = (uint32_t)x & pmask;
            vo[p] = sm.vals[q];
            if (!FLAGS) {
                uint32_t q_;
                ko[p] = (K)onchip_key(sm, f, x, &q_);
            }
            if (FLAGS) {
                const unsigned long long y = sm.cs[p ? p - 1 : 0u];
                bool differs = p == 0 || (x ^ y) > pmask;
                if constexpr (sizeof(K) == 8) {
                    if (f.drop && !differs) differs = sm.lo[q] != sm.lo[(uint32_t)y & pmask];
                }
                fo[p] = differs;
            }
        }
    }
    group_sync<NT>();
}

// CTA per segment.  1024 threads per SM for every tier (64 registers a thread).
template <typename K, int NT, int IT, bool FLAGS>
__global__ void __launch_bounds__(NT, 1024 / NT)
block_sort_kernel(Bufs<K> b, const uint2 *list, const uint32_t *d_count)
{
    kernel_prologue();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const uint32_t count = *d_count;
    for (uint32_t e = blockIdx.x; e < count; e += gridDim.x) {
        const uint2 ent = list[e];
        onchip_sort<K, NT, IT, FLAGS>(*reinterpret_cast<OnchipSmem<K, NT, IT> *>(smem_raw), b, ent.x, ent.y & 0xFFFFu,
                               (ent.y >> 24) & 3u);
    }
}

// Warp per segment, kWarpsA warps a CTA.  The grid is what fits at once.
constexpr int kWarpsA = 4;
constexpr int warp_ctas_per_sm(int it) { return it <= 4 ? 10 : 7; }
template <typename K, int IT, bool FLAGS>
__global__ void __launch_bounds__(kWarpsA * 32, warp_ctas_per_sm(IT))
warp_sort_kernel(Bufs<K> b, const uint2 *list, const uint32_t *d_count)
{
    kernel_prologue();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    OnchipSmem<K, 32, IT> &sm = reinterpret_cast<OnchipSmem<K, 32, IT> *>(smem_raw)[threadIdx.x >> 5];
    const uint32_t count = *d_count;
    for (uint32_t e = blockIdx.x * kWarpsA + (threadIdx.x >> 5); e < count; e += gridDim.x * kWarpsA) {
        const uint2 ent = list[e];
        onchip_sort<K, 32, IT, FLAGS>(sm, b, ent.x, ent.y & 0xFFFFu, (ent.y >> 24) & 3u);
    }
}

// Thread-per-segment sort of tiny segments (2..kCapT rows): the rows sit in
// registers and an odd-even transposition network of N rounds sorts them.
// It swaps only strictly inverted neighbours, so equal keys keep their order
// (stable); the padding slots hold the largest key and stay behind the rows.
template <typename K, int N, bool FLAGS>
__device__ __forceinline__ void sort_tiny(const Bufs<K> &b, uint32_t start, uint32_t len, uint32_t src)
{
    K k[N];
    uint32_t v[N];
#pragma unroll
    for (int i = 0; i < N; ++i) {
        k[i] = ~K(0);
        v[i] = 0;
        if (i < (int)len) load_kv(b, src, (uint64_t)start + i, k[i], v[i]);
    }
#pragma unroll
    for (int r = 0; r < N; ++r) {
#pragma unroll
        for (int i = r & 1; i + 1 < N; i += 2) {
            if (k[i] > k[i + 1]) {
                const K tk = k[i];
                k[i] = k[i + 1];
                k[i + 1] = tk;
                const uint32_t tv = v[i];
                v[i] = v[i + 1];
                v[i + 1] = tv;
            }
        }
    }
#pragma unroll
    for (int i = 0; i < N; ++i) {
        if (i < (int)len) {
            if (!FLAGS) b.k0[(uint64_t)start + i] = k[i];
            b.v0[(uint64_t)start + i] = v[i];
            if (FLAGS) b.flags[(uint64_t)start + i] = i == 0 || k[i] != k[i > 0 ? i - 1 : 0];
        }
    }
}

template <typename K, int NMAX, bool FLAGS>
__global__ void __launch_bounds__(256) thread_sort_kernel(Bufs<K> b, const uint2 *list, const uint32_t *d_count)
{
    kernel_prologue();
    const uint32_t count = *d_count;
    for (uint32_t e = blockIdx.x * blockDim.x + threadIdx.x; e < count; e += gridDim.x * blockDim.x) {
        const uint2 ent = list[e];
        const uint32_t start = ent.x;
        const uint32_t len = ent.y & 0xFFFFu;
        const uint32_t src = (ent.y >> 24) & 3u;
        if constexpr (NMAX > 16) {
            sort_tiny<K, NMAX, FLAGS>(b, start, len, src);
        } else {
            if (len <= 2) sort_tiny<K, 2, FLAGS>(b, start, len, src);
            else if (len <= 4) sort_tiny<K, 4, FLAGS>(b, start, len, src);
            else if (len <= 8) sort_tiny<K, 8, FLAGS>(b, start, len, src);
            else sort_tiny<K, 16, FLAGS>(b, start, len, src);
        }
    }
}

// A row of a segment that needs no sorting: to BUF0 unless it is there, and its
// flag (the segment's keys are equal).
template <typename K>
__device__ __forceinline__ void copy_row(const Bufs<K> &b, const LargeSeg &sg, uint64_t r)
{
    if ((sg.src & 3u) != kSrcBuf0) {
        K k;
        uint32_t v;
        load_kv(b, sg.src & 3u, r, k, v);
        if (b.write_keys) b.k0[r] = k;
        b.v0[r] = v;
    }
    if (b.flags) b.flags[r] = r == sg.start;
}

// Segments that need no sorting but sit outside BUF0 (or lack their flags): one
// warp per entry.
template <typename K>
__global__ void __launch_bounds__(256) copy_kernel(Bufs<K> b, const LargeSeg *list, const uint32_t *d_count)
{
    kernel_prologue();
    const uint32_t count = *d_count;
    const int lane = threadIdx.x & 31;
    const uint32_t nwarps = gridDim.x * (blockDim.x / 32);
    for (uint32_t e = blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5); e < count; e += nwarps) {
        const LargeSeg sg = list[e];
        for (uint32_t i = lane; i < sg.len; i += 32) copy_row(b, sg, (uint64_t)sg.start + i);
    }
}

// Large segments that only need to reach BUF0: tiles of kCopySplit rows
// spread over the whole grid (tile -> segment by binary search).
template <typename K>
__global__ void __launch_bounds__(256) copy_tiles_kernel(Bufs<K> b, const LargeSeg *list, const uint32_t *d_count,
                                                         const uint32_t *tile_prefix)
{
    kernel_prologue();
    const uint32_t count = *d_count;
    if (count == 0) return;
    const uint32_t T = tile_prefix[count];
    for (uint32_t t = blockIdx.x; t < T; t += gridDim.x) {
        const uint32_t s = find_segment_warp(tile_prefix, count, t);
        const LargeSeg sg = list[s];
        const uint64_t beg = (uint64_t)sg.start + (uint64_t)(t - tile_prefix[s]) * kCopySplit;
        const uint64_t end = min((uint64_t)sg.start + sg.len, beg + kCopySplit);
        for (uint64_t r = beg + threadIdx.x; r < end; r += blockDim.x) copy_row(b, sg, r);
    }
}

#define FMCS_LAUNCH_CHECK(what)                                         \
    do {                                                                \
        cudaError_t e_ = cudaGetLastError();                            \
        if (e_ != cudaSuccess) return cuda_fail(ctx, e_, what);          \
    } while (0)

template <typename K, int RANK, int IT>
int sort_segments_t(fmcs_ctx *ctx, const SortArgs &a)
{
    const uint64_t n = a.n;
    cudaStream_t st = ctx->stream;
    // buffers
    Bufs<K> b;
    b.ext_bank = (const K *)a.bank;
    b.ext_order = a.order_in;
    b.flags = a.flags;
    b.write_keys = a.flags == nullptr;
    void *p = nullptr;
    int rc;
    if (a.keys_out) {
        b.k0 = (K *)a.keys_out;
    } else {
        if ((rc = ws_get(ctx, kSlotKeys0, n * sizeof(K), &p))) return rc;
        b.k0 = (K *)p;
    }
    b.v0 = a.order_out;
    if ((rc = ws_get(ctx, kSlotKeys1, n * sizeof(K), &p))) return rc;
    b.k1 = (K *)p;
    if ((rc = ws_get(ctx, kSlotVals1, n * sizeof(uint32_t), &p))) return rc;
    b.v1 = (uint32_t *)p;

    // lists (capacities are bounds on disjoint segments of each tier's minimum size)
    const uint32_t local_max = std::max<uint32_t>(kCapA, std::min<uint32_t>(ctx->local_max, kCapLocal));
    const SortListCaps caps = sort_list_caps(n, local_max, a.key_bits);
    const uint64_t cap_large = caps.large;
    const uint64_t cap_t = n / 2 + 2, cap_t32 = n / (kCapT + 1) + 2, cap_a = n / (kCapT + 1) + 2;
    const uint64_t cap_a2 = n / (kCapA + 1) + 2, cap_b1 = n / (kCapA2 + 1) + 2;
    const uint64_t cap_b2 = n / (kCapB1 + 1) + 2;
    const uint64_t cap_c1 = n / (kCapB2 + 1) + 2, cap_c1b = n / (kCapC1 + 1) + 2, cap_c2 = n / (kCapC1b + 1) + 2;
    const uint64_t cap_c3 = n / (kCapC2 + 1) + 2;
    LargeSeg *large[2];
    if ((rc = ws_get(ctx, kSlotLarge0, cap_large * sizeof(LargeSeg), &p))) return rc;
    large[0] = (LargeSeg *)p;
    if ((rc = ws_get(ctx, kSlotLarge1, cap_large * sizeof(LargeSeg), &p))) return rc;
    large[1] = (LargeSeg *)p;
    Lists lists;
    {
        const size_t e = sizeof(uint2);
        if ((rc = ws_get(ctx, kSlotLocalA,
                         carve_total({cap_t * e, cap_t32 * e, cap_a * e, cap_a2 * e, cap_b1 * e, cap_b2 * e, cap_c1 * e,
                                      cap_c1b * e, cap_c2 * e, cap_c3 * e}),
                         &p)))
            return rc;
        Carver cv(p);
        lists.t = cv.take<uint2>(cap_t);
        lists.t32 = cv.take<uint2>(cap_t32);
        lists.a = cv.take<uint2>(cap_a);
        lists.a2 = cv.take<uint2>(cap_a2);
        lists.cap_t32 = sizeof(K) <= 4 ? kCapT32 : 0;
        lists.b1 = cv.take<uint2>(cap_b1);
        lists.b2 = cv.take<uint2>(cap_b2);
        lists.c1 = cv.take<uint2>(cap_c1);
        lists.c1b = cv.take<uint2>(cap_c1b);
        lists.c2 = cv.take<uint2>(cap_c2);
        lists.c3 = cv.take<uint2>(cap_c3);
        if ((rc = ws_get(ctx, kSlotLocalC, carve_total({caps.copy * sizeof(LargeSeg), caps.copy_large * sizeof(LargeSeg)}),
                         &p)))
            return rc;
        Carver cc(p);
        lists.copy = cc.take<LargeSeg>(caps.copy);
        lists.copy_large = cc.take<LargeSeg>(caps.copy_large);
        lists.local_max = local_max;
        lists.flags = a.flags;
    }
    // (a segment's chunks <= its rows / chunk_rows + 1)
    LevelRefs lr{};
    lr.large[0] = large[0];
    lr.large[1] = large[1];
    lr.chunk_rows = msd_chunk_rows(ctx, n);
    lr.max_chunks = (uint32_t)(n / lr.chunk_rows);
    const uint64_t cap_chunks = n / lr.chunk_rows + cap_large + 1;
    const uint64_t cap_super = super_rows_max(cap_chunks, cap_large);
    const uint64_t cap_long = 2 * (cap_chunks / kSuper) + 2;   // ceil(c / kSuper) <= 2 c / kSuper for c > kSuper
    const size_t row = kRadix * sizeof(uint32_t);
    if ((rc = ws_get(ctx, kSlotSegHist,
                     carve_total({cap_chunks * row, cap_super * row, cap_super * row, cap_chunks * sizeof(Chunk),
                                  cap_long * sizeof(uint2)}),
                     &p)))
        return rc;
    {
        Carver cv(p);
        lr.hist = cv.take<uint32_t>(cap_chunks * kRadix);
        lr.super[0] = cv.take<uint32_t>(cap_super * kRadix);
        lr.super[1] = cv.take<uint32_t>(cap_super * kRadix);
        lr.work = cv.take<Chunk>(cap_chunks);
        lr.long_rows = cv.take<uint2>(cap_long);
    }
    uint32_t *tile_prefix;   // of the large copies
    if ((rc = ws_get(ctx, kSlotTilePrefix, carve_total({(caps.copy_large + 1) * sizeof(uint32_t),
                                                        (cap_large + 1) * sizeof(uint32_t)}), &p)))
        return rc;
    {
        Carver cv(p);
        tile_prefix = cv.take<uint32_t>(caps.copy_large + 1);
        lr.chunk_prefix = cv.take<uint32_t>(cap_large + 1);
    }
    uint32_t *ctr;
    if ((rc = ws_get(ctx, kSlotCounters, 4096, &p))) return rc;
    ctr = (uint32_t *)p + 64;   // words 0..63 belong to other kernels
    cudaMemsetAsync(ctr, 0, kCtrWords * sizeof(uint32_t), st);
    lr.ctr = ctr;
    lr.dev_level = 1;
    lr.top_hist = a.seg_start ? nullptr : a.top_hist;
    lr.gathered = a.order_in && a.order_in == a.order_out;

    const int sms = ctx->num_sms;
    // classification of the initial segments
    {
        const uint32_t *seg_start = a.seg_start;
        const uint32_t *d_nseg = a.d_nseg;
        unsigned grid = seg_start ? (unsigned)std::min<uint64_t>((a.nseg_host + 255) / 256 + 1, (uint64_t)sms * 16)
                                  : 1u;
        if (seg_start && a.nseg_host == 0) grid = (unsigned)sms * 16;
        if (a.d_in_order) grid = std::max(grid, (unsigned)sms * 4);   // (it may copy every row)
        { LaunchScope ls_(ctx, "classify");
            launch_k(classify_kernel<K>, grid, 256, 0, st, b, seg_start, d_nseg, n, a.key_bits, ctr, large[0], lists,
                     lr.top_hist, a.d_key_bits, a.d_in_order,
                     a.skip_single && a.order_in == a.order_out, a.flags && a.mark_starts);
        }
        FMCS_LAUNCH_CHECK("classify");
    }
    // The host's copy of the counters when an eager call
    // has read them back after the last routing of segments to the tiers.
    bool tiers_known = false;
    uint32_t *hctr = ctx->h_small + kHostCounters;
    if (!a.fixed_launches && !a.seg_start && (!a.d_key_bits || a.d_in_order) && n <= (uint64_t)local_max) {
        // A round 0 that fits one tier (a hash round's clustering, or a plan of too
        // many banks or slices for one launch): the host routes it as classify
        // does.  (Rows with no key bits left are in order, and classify copies
        // those.  A hash plan of 1,000 rows: 108 us with every tier launched, 81 so.)
        uint32_t *w = hctr;
        for (int i = 0; i < kCtrWords; ++i) w[i] = 0;
        const uint32_t len = (uint32_t)n;
        if (len > 1) {
            const int which = len <= (uint32_t)kCapT ? kCtrLocalT
                              : len <= lists.cap_t32 ? kCtrLocalT32
                              : len <= (uint32_t)kCapA ? kCtrLocalA
                              : len <= (uint32_t)kCapA2 ? kCtrLocalA2
                              : len <= (uint32_t)kCapB1 ? kCtrLocalB1
                              : len <= (uint32_t)kCapB2 ? kCtrLocalB2
                              : len <= (uint32_t)kCapC1 ? kCtrLocalC1
                              : len <= (uint32_t)kCapC1b ? kCtrLocalC1b
                              : len <= (uint32_t)kCapC2 ? kCtrLocalC2 : kCtrLocalC3;
            w[which] = 1;
        }
        tiers_known = true;
    }
    if (!a.fixed_launches && a.seg_start) {
        // how many segments each way of sorting them got
        const uint32_t seq = ++ctx->read_backs;
        if ((rc = launch_publish_counters(ctx, ctr, seq))) return rc;
        if ((rc = wait_counters(ctx, seq, "sort: segment counts"))) return rc;
        tiers_known = true;
    }
    // MSD levels
    const int levels = (int)((a.key_bits + kRadixBits - 1) / kRadixBits);
    const size_t msd_smem = sizeof(MsdSmem<K, IT>);
    if ((rc = raise_smem(ctx, (const void *)msd_scatter_kernel<K, RANK, IT>, msd_smem))) return rc;
    if (n > (uint64_t)local_max) {
        // Host-known count of the level's large segments (exact unless the
        // caller asked for a fixed launch sequence, e.g. for graph capture).
        uint32_t nlarge = a.fixed_launches || !a.seg_start ? 1u : hctr[kCtrLarge0];
        const unsigned scatter_grid = sms * msd_ctas_per_sm(IT);
        int host_lvl = 0;   // the level being launched, for the eager read-back
        // one level: the same four launches for every level (the level index
        // lives on the device)
        auto level = [&](cudaStream_t s, cudaGraphConditionalHandle more, bool read_back) -> int {
            { LaunchScope ls_(ctx, "tile_prefix");
                launch_k(level_prefix_kernel, 1, 1024, 0, s, lr);
            }
            if (!(lr.top_hist && host_lvl == 0 && read_back)) {
                // (inside a graph the launch stays and returns at once on level 0)
                LaunchScope ls_(ctx, "msd_hist");
                launch_k(msd_hist_kernel<K>, sms * kHistCtas, kNtM, 0, s, b, lr);
            }
            { LaunchScope ls_(ctx, "msd_plan");
                launch_k(msd_plan_kernel, sms * 8, kPlanThreads, 0, s, lr, lists, true);
            }
            {
                LaunchScope ls_(ctx, "msd_scatter");
                const uint32_t seq = read_back ? ++ctx->read_backs : 0u;
                launch_k(msd_scatter_kernel<K, RANK, IT>, scatter_grid, kNtM, msd_smem, s, b, lr, more,
                         (uint32_t)levels, read_back ? ctx->h_small : (uint32_t *)nullptr, seq);
                FMCS_LAUNCH_CHECK("msd level");
                if (read_back) {
                    if ((rc = wait_counters(ctx, seq, "sort: level counts"))) return rc;
                    // algorithmic bytes: every moved row is read from the level's
                    // source (the round's bank, through the order when there is
                    // one, at level 0; the work buffers after) and written once
                    const double moved = (double)hctr[kCtrMoved];
                    const double rd = host_lvl == 0 ? (double)sizeof(K) + (b.ext_order ? 4.0 : 0.0)
                                                    : (double)sizeof(K) + 4.0;
                    ls_.set_units(moved);
                    ls_.set_bytes(moved * (rd + (double)sizeof(K) + 4.0));
                }
            }
            FMCS_LAUNCH_CHECK("msd level");
            return FMCS_OK;
        };
        cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
        if (a.fixed_launches && cudaStreamIsCapturing(st, &cap) == cudaSuccess && cap == cudaStreamCaptureStatusActive) {
            // graph capture: the levels are one WHILE node whose body is one
            // level; each level's scatter decides whether another follows
            if ((rc = capture_while(ctx, st, [&](cudaStream_t s, cudaGraphConditionalHandle h) {
                     return level(s, h, false);
                 })))
                return rc;
        } else {
            for (int lvl = 0; lvl < levels && nlarge > 0; ++lvl) {
                host_lvl = lvl;
                if ((rc = level(st, 0, !a.fixed_launches))) return rc;
                if (!a.fixed_launches) {
                    nlarge = hctr[kCtrLarge0 + ((uint32_t)(lvl + 1) & 1u)];
                    tiers_known = true;
                }
            }
        }
    }
    // local tiers (they write flags or keys)
    const bool fo = a.flags != nullptr;
    const size_t smem_a = kWarpsA * sizeof(OnchipSmem<K, 32, kItA>);
    const size_t smem_a2 = kWarpsA * sizeof(OnchipSmem<K, 32, kItA2>);
    const size_t smem_b1 = sizeof(OnchipSmem<K, kNtB1, kItB1>);
    const size_t smem_b2 = sizeof(OnchipSmem<K, kNtB2, kItB2>);
    const size_t smem_c1 = sizeof(OnchipSmem<K, kNtC1, kItC1>);
    const size_t smem_c1b = sizeof(OnchipSmem<K, kNtC1b, kItC1b>);
    const size_t smem_c2 = sizeof(OnchipSmem<K, kNtC2, kItC2>);
    const size_t smem_c3 = sizeof(OnchipSmem<K, kNtC3, kItC3>);
    auto set_smem2 = [&](auto *k0, auto *k1, size_t bytes) -> int {
        return raise_smem(ctx, (const void *)(fo ? k1 : k0), bytes);
    };
    if ((rc = set_smem2(warp_sort_kernel<K, kItA, false>, warp_sort_kernel<K, kItA, true>, smem_a))) return rc;
    if ((rc = set_smem2(warp_sort_kernel<K, kItA2, false>, warp_sort_kernel<K, kItA2, true>, smem_a2))) return rc;
    if ((rc = set_smem2(block_sort_kernel<K, kNtB1, kItB1, false>, block_sort_kernel<K, kNtB1, kItB1, true>, smem_b1))) return rc;
    if ((rc = set_smem2(block_sort_kernel<K, kNtB2, kItB2, false>, block_sort_kernel<K, kNtB2, kItB2, true>, smem_b2))) return rc;
    if ((rc = set_smem2(block_sort_kernel<K, kNtC1, kItC1, false>, block_sort_kernel<K, kNtC1, kItC1, true>, smem_c1))) return rc;
    if ((rc = set_smem2(block_sort_kernel<K, kNtC1b, kItC1b, false>, block_sort_kernel<K, kNtC1b, kItC1b, true>, smem_c1b))) return rc;
    if ((rc = set_smem2(block_sort_kernel<K, kNtC2, kItC2, false>, block_sort_kernel<K, kNtC2, kItC2, true>, smem_c2))) return rc;
    if ((rc = set_smem2(block_sort_kernel<K, kNtC3, kItC3, false>, block_sort_kernel<K, kNtC3, kItC3, true>, smem_c3))) return rc;
    // Each tier's launch, with the counter word of its list.  An eager call
    // that knows the lists' sizes from its last read-back (tiers_known) does
    // not launch a tier whose list is empty.  A captured graph launches every
    // tier (an empty one returns at once): one conditional node per tier cost
    // more on replay than the empty launches it saved.
    struct Tier {
        int word;
        std::function<void(cudaStream_t, bool)> launch;   // bool: may begin while its predecessor finishes
    };
    std::vector<Tier> tiers;
    // CTAs of a tier: enough for its list where the host knows its length (a
    // CTA that finds no segment still takes its share of an SM from the other
    // streams until its predecessor is done), else all that are resident.
    // (90,001 rows in two banks: 180 -> 170 us a call; five instances of 128 K
    // to 512 K rows: 210 -> 189 us)
    auto ctas = [&](int word, int resident, int segs_per_cta) -> int {
        if (!tiers_known) return resident;
        const uint32_t want = (hctr[word] + segs_per_cta - 1) / segs_per_cta;
        return want < (uint32_t)resident ? (int)want : resident;
    };
    tiers.push_back({kCtrLocalT, [&](cudaStream_t s, bool early) {
        LaunchScope ls_(ctx, "thread_sort");
        launch_on(early, fo ? thread_sort_kernel<K, 16, true> : thread_sort_kernel<K, 16, false>, ctas(kCtrLocalT, sms * 8, 256), 256, 0, s, b, lists.t, &ctr[kCtrLocalT]);
    }});
    if constexpr (sizeof(K) <= 4) {
        tiers.push_back({kCtrLocalT32, [&](cudaStream_t s, bool early) {
            LaunchScope ls_(ctx, "thread_sort_32");
            launch_on(early, fo ? thread_sort_kernel<K, 32, true> : thread_sort_kernel<K, 32, false>, ctas(kCtrLocalT32, sms * 8, 256), 256, 0, s, b, lists.t32, &ctr[kCtrLocalT32]);
        }});
    }
    tiers.push_back({kCtrLocalA, [&](cudaStream_t s, bool early) {
        LaunchScope ls_(ctx, "warp_sort");
        launch_on(early, fo ? warp_sort_kernel<K, kItA, true> : warp_sort_kernel<K, kItA, false>, ctas(kCtrLocalA, sms * warp_ctas_per_sm(kItA), kWarpsA), kWarpsA * 32, smem_a, s, b, lists.a, &ctr[kCtrLocalA]);
    }});
    tiers.push_back({kCtrLocalA2, [&](cudaStream_t s, bool early) {
        LaunchScope ls_(ctx, "warp_sort_256");
        launch_on(early, fo ? warp_sort_kernel<K, kItA2, true> : warp_sort_kernel<K, kItA2, false>, ctas(kCtrLocalA2, sms * warp_ctas_per_sm(kItA2), kWarpsA), kWarpsA * 32, smem_a2, s, b, lists.a2, &ctr[kCtrLocalA2]);
    }});
    tiers.push_back({kCtrLocalB1, [&](cudaStream_t s, bool early) {
        LaunchScope ls_(ctx, "block_sort_512");
        launch_on(early, fo ? block_sort_kernel<K, kNtB1, kItB1, true> : block_sort_kernel<K, kNtB1, kItB1, false>, ctas(kCtrLocalB1, sms * (1024 / kNtB1), 1), kNtB1, smem_b1, s, b, lists.b1,
                  &ctr[kCtrLocalB1]);
    }});
    tiers.push_back({kCtrLocalB2, [&](cudaStream_t s, bool early) {
        LaunchScope ls_(ctx, "block_sort_1024");
        launch_on(early, fo ? block_sort_kernel<K, kNtB2, kItB2, true> : block_sort_kernel<K, kNtB2, kItB2, false>, ctas(kCtrLocalB2, sms * (1024 / kNtB2), 1), kNtB2, smem_b2, s, b, lists.b2,
                 &ctr[kCtrLocalB2]);
    }});
    tiers.push_back({kCtrLocalC1, [&](cudaStream_t s, bool early) {
        LaunchScope ls_(ctx, "block_sort_2048");
        launch_on(early, fo ? block_sort_kernel<K, kNtC1, kItC1, true> : block_sort_kernel<K, kNtC1, kItC1, false>, ctas(kCtrLocalC1, sms * (1024 / kNtC1), 1), kNtC1, smem_c1, s, b, lists.c1,
                 &ctr[kCtrLocalC1]);
    }});
    tiers.push_back({kCtrLocalC1b, [&](cudaStream_t s, bool early) {
        LaunchScope ls_(ctx, "block_sort_2304");
        launch_on(early, fo ? block_sort_kernel<K, kNtC1b, kItC1b, true> : block_sort_kernel<K, kNtC1b, kItC1b, false>, ctas(kCtrLocalC1b, sms * (1024 / kNtC1b), 1), kNtC1b, smem_c1b, s, b, lists.c1b,
                 &ctr[kCtrLocalC1b]);
    }});
    tiers.push_back({kCtrLocalC2, [&](cudaStream_t s, bool early) {
        LaunchScope ls_(ctx, "block_sort_4096");
        launch_on(early, fo ? block_sort_kernel<K, kNtC2, kItC2, true> : block_sort_kernel<K, kNtC2, kItC2, false>, ctas(kCtrLocalC2, sms * (1024 / kNtC2), 1), kNtC2, smem_c2, s, b, lists.c2,
                 &ctr[kCtrLocalC2]);
    }});
    tiers.push_back({kCtrLocalC3, [&](cudaStream_t s, bool early) {
        LaunchScope ls_(ctx, "block_sort_8192");
        launch_on(early, fo ? block_sort_kernel<K, kNtC3, kItC3, true> : block_sort_kernel<K, kNtC3, kItC3, false>, ctas(kCtrLocalC3, sms * (1024 / kNtC3), 1), kNtC3, smem_c3, s, b, lists.c3,
                 &ctr[kCtrLocalC3]);
    }});
    tiers.push_back({kCtrCopy, [&](cudaStream_t s, bool early) {
        LaunchScope ls_(ctx, "copy");
        launch_on(early, copy_kernel<K>, sms * 4, 256, 0, s, b, lists.copy, &ctr[kCtrCopy]);
    }});
    tiers.push_back({kCtrCopyLarge, [&](cudaStream_t s, bool) {
        {
            LaunchScope ls_(ctx, "tile_prefix");
            launch_k(tile_prefix_kernel, 1, 1024, 0, s, lists.copy_large, &ctr[kCtrCopyLarge], tile_prefix,
                     &ctr[kCtrCopyTile], kCopySplit);
        }
        LaunchScope ls_(ctx, "copy_tiles");
        launch_k(copy_tiles_kernel<K>, sms * 8, 256, 0, s, b, lists.copy_large, &ctr[kCtrCopyLarge], tile_prefix);
    }});
    // The tiers' segments are disjoint: the tiers up to the 2048-row one run
    // on the context's stream, the larger ones and the copies on its second
    // stream at the same time, so that a tier with few segments (one wave of
    // one segment per CTA, latency-bound) overlaps a busy one.  While
    // profiling, every tier stays on the context's stream (one at a time,
    // each timed alone).
    auto wanted = [&](const Tier &t) { return !tiers_known || hctr[t.word] > 0; };
    // A tier with enough segments to fill the GPU waits for its predecessor to
    // leave the SMs.  CTAs that move in while the predecessor's are still
    // resident split up the shared memory between them, and the last CTA of
    // each SM no longer fits: it runs as a second wave, with a whole CTA's
    // share of the segments (40M-row wide ORDER BY: the 2048-row tier 734 us
    // instead of 484).  With few segments the early start saves 3 us a tier.
    auto early = [&](const Tier &t) {
        return tiers_known ? hctr[t.word] <= (uint32_t)sms : n < (uint64_t)kCapLocal * 32u;
    };
    size_t split = 0;
    while (split < tiers.size() && tiers[split].word != kCtrLocalC1b) ++split;
    bool two = !ctx->prof_on;
    if (two) {
        bool a = false, bb = false;
        for (size_t i = 0; i < tiers.size(); ++i) (i < split ? a : bb) |= wanted(tiers[i]);
        two = a && bb;
    }
    if (two) {
        if ((rc = fork_par(ctx, st))) return rc;
        for (size_t i = 0; i < tiers.size(); ++i)
            if (wanted(tiers[i])) tiers[i].launch(i < split ? st : ctx->par, early(tiers[i]));
        if ((rc = join_par(ctx, st))) return rc;
    } else {
        for (const Tier &t : tiers)
            if (wanted(t)) t.launch(st, early(t));
    }
    FMCS_LAUNCH_CHECK("local tiers");
    return FMCS_OK;
}

// ---------------------------------------------------------------------------
// Full-array LSD radix sort (the plain comparator path: no segments, no
// binning).  One pass per 8 key bits, each pass the MSD level kernels applied
// to a single segment [0, n) with the digit at bits [shift-8, shift).  Passes
// where every row has the same digit are skipped on the device, so the buffer
// holding the result is tracked on the device and a final copy puts it in
// BUF0.
// ---------------------------------------------------------------------------
__global__ void lsd_set_pass_kernel(LargeSeg *seg, uint32_t *nseg, uint32_t n, uint32_t shift, int first)
{
    kernel_prologue();
    if (threadIdx.x == 0) {
        uint32_t src = kSrcBuf0;
        if (!first) {
            const LargeSeg prev = seg[0];
            src = (prev.src & kSkipBit) ? (prev.src & 3u) : ((prev.src & 3u) == kSrcBuf1 ? kSrcBuf0 : kSrcBuf1);
        }
        seg[0] = LargeSeg{0, n, shift, src};
        *nseg = 1;
    }
}

template <typename K>
__global__ void lsd_finalize_kernel(Bufs<K> b, const LargeSeg *seg, uint64_t n)
{
    kernel_prologue();
    const LargeSeg last = seg[0];
    const uint32_t where = (last.src & kSkipBit) ? (last.src & 3u) : ((last.src & 3u) == kSrcBuf1 ? kSrcBuf0 : kSrcBuf1);
    if (where != kSrcBuf1) return;
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        b.k0[i] = b.k1[i];
        b.v0[i] = b.v1[i];
    }
}

template <typename K, int RANK, int IT>
int lsd_sort_full_t(fmcs_ctx *ctx, void *keys, uint32_t *vals, uint64_t n, uint32_t bits)
{
    cudaStream_t st = ctx->stream;
    int rc;
    void *p;
    Bufs<K> b;
    b.k0 = (K *)keys;
    b.v0 = vals;
    b.ext_bank = nullptr;
    b.ext_order = nullptr;
    b.flags = nullptr;
    b.write_keys = 1;
    if ((rc = ws_get(ctx, kSlotKeys1, n * sizeof(K), &p))) return rc;
    b.k1 = (K *)p;
    if ((rc = ws_get(ctx, kSlotVals1, n * sizeof(uint32_t), &p))) return rc;
    b.v1 = (uint32_t *)p;
    LargeSeg *seg;
    if ((rc = ws_get(ctx, kSlotLarge0, sizeof(LargeSeg) * 2, &p))) return rc;
    seg = (LargeSeg *)p;
    // one segment [0, n), re-set before every pass; level buffers of set 0
    LevelRefs lr{};
    lr.large[0] = seg;
    lr.large[1] = seg + 1;
    // (a pass's tiles have IT rows a thread whatever msd_items is.  As long as they
    // all run at once a chunk is one tile: chunks of two make every CTA take them
    // one after the other (300,000 rows of 50-bit keys: 284 us, one-tile chunks 217; 1.2M
    // 311 and 270; 2M 330 and 343, 8M 861 and 889).)
    const uint64_t tile = (uint64_t)kNtM * IT;
    lr.chunk_rows = n <= tile * ctx->num_sms * msd_ctas_per_sm(IT) ? (uint32_t)tile : msd_chunk_rows(ctx, n);
    lr.max_chunks = (uint32_t)(n / lr.chunk_rows);
    const uint64_t chunks = (n - 1) / lr.chunk_rows + 1, supers = super_rows_max(chunks, 1);
    const size_t row = kRadix * sizeof(uint32_t);
    if ((rc = ws_get(ctx, kSlotSegHist,
                     carve_total({chunks * row, supers * row, chunks * sizeof(Chunk),
                                  (chunks / kSuper + 1) * sizeof(uint2)}),
                     &p)))
        return rc;
    {
        Carver cv(p);
        lr.hist = cv.take<uint32_t>(chunks * kRadix);
        lr.super[0] = cv.take<uint32_t>(supers * kRadix);
        lr.work = cv.take<Chunk>(chunks);
        lr.long_rows = cv.take<uint2>(chunks / kSuper + 1);
    }
    if ((rc = ws_get(ctx, kSlotTilePrefix, 2 * sizeof(uint32_t), &p))) return rc;
    lr.chunk_prefix = (uint32_t *)p;
    uint32_t *ctr;
    if ((rc = ws_get(ctx, kSlotCounters, 4096, &p))) return rc;
    ctr = (uint32_t *)p + 64;
    lr.ctr = ctr;
    const size_t msd_smem = sizeof(MsdSmem<K, IT>);
    if ((rc = raise_smem(ctx, (const void *)msd_scatter_kernel<K, RANK, IT>, msd_smem))) return rc;
    const int sms = ctx->num_sms;
    Lists none{};
    int pass = 0;
    for (uint32_t lo = 0; lo < bits; lo += kRadixBits, ++pass) {
        const uint32_t shift = std::min(bits, lo + kRadixBits);
        { LaunchScope ls_(ctx, "lsd_set_pass");
            launch_k(lsd_set_pass_kernel, 1, 32, 0, st, seg, &ctr[kCtrLarge0], (uint32_t)n, shift, pass == 0);
        }
        { LaunchScope ls_(ctx, "tile_prefix");
            launch_k(level_prefix_kernel, 1, 1024, 0, st, lr);
        }
        { LaunchScope ls_(ctx, "msd_hist");
            launch_k(msd_hist_kernel<K>, sms * kHistCtas, kNtM, 0, st, b, lr);
        }
        { LaunchScope ls_(ctx, "msd_plan");
            launch_k(msd_plan_kernel, sms, kPlanThreads, 0, st, lr, none, false);
        }
        { LaunchScope ls_(ctx, "msd_scatter");
            launch_k(msd_scatter_kernel<K, RANK, IT>, sms * msd_ctas_per_sm(IT), kNtM, msd_smem, st, b, lr,
                     (cudaGraphConditionalHandle)0, 1u, (uint32_t *)nullptr, 0u);
        }
        FMCS_LAUNCH_CHECK("lsd pass");
    }
    if (pass > 0) {
        LaunchScope ls_(ctx, "lsd_finalize");
        launch_k(lsd_finalize_kernel<K>, sms * 8, 256, 0, st, b, seg, n);
    }
    FMCS_LAUNCH_CHECK("lsd finalize");
    return FMCS_OK;
}

}  // namespace

uint32_t msd_chunk_rows(const fmcs_ctx *ctx, uint64_t n)
{
    uint64_t rows = (uint64_t)kNtM * (ctx->msd_items >= 16 ? 16u : 8u);
    while (rows * 2 * kChunksWanted <= n) rows *= 2;
    return (uint32_t)rows;
}

int lsd_sort_full(fmcs_ctx *ctx, void *keys, uint32_t key_bytes, uint32_t *vals, uint64_t n, uint32_t bits)
{
    if (n <= 1 || bits == 0) return FMCS_OK;
    switch (key_bytes) {
    case 4: return lsd_sort_full_t<uint32_t, kRankMatch, 8>(ctx, keys, vals, n, bits);
    case 8: return lsd_sort_full_t<uint64_t, kRankMatch, 8>(ctx, keys, vals, n, bits);
    case 2: return lsd_sort_full_t<uint16_t, kRankMatch, 8>(ctx, keys, vals, n, bits);
    default: return set_error(ctx, FMCS_E_INVAL, "lsd sort: key bytes must be 2, 4 or 8");
    }
}

template <typename K>
static int sort_dispatch(fmcs_ctx *ctx, const SortArgs &a)
{
    const bool big = ctx->msd_items >= 16;
    if (ctx->rank_mode == 2)
        return big ? sort_segments_t<K, kRankOr, 16>(ctx, a) : sort_segments_t<K, kRankOr, 8>(ctx, a);
    if (ctx->rank_mode)
        return big ? sort_segments_t<K, kRankBallot, 16>(ctx, a) : sort_segments_t<K, kRankBallot, 8>(ctx, a);
    return big ? sort_segments_t<K, kRankMatch, 16>(ctx, a) : sort_segments_t<K, kRankMatch, 8>(ctx, a);
}

int sort_segments(fmcs_ctx *ctx, const SortArgs &a)
{
    if (a.n == 0) return FMCS_OK;
    if (a.flags && a.d_in_order) return set_error(ctx, FMCS_E_INVAL, "sort: rows that may be in order have no flags");
    if (a.key_bits == 0 || a.key_bits > 8 * a.bank_bytes)
        return set_error(ctx, FMCS_E_INVAL, "sort: key_bits must be in 1..8*bank_bytes");
    switch (a.bank_bytes) {
    case 2: return sort_dispatch<uint16_t>(ctx, a);
    case 4: return sort_dispatch<uint32_t>(ctx, a);
    case 8: return sort_dispatch<uint64_t>(ctx, a);
    default: return set_error(ctx, FMCS_E_INVAL, "sort: bank_bytes must be 2, 4 or 8");
    }
}

}  // namespace fmcs
