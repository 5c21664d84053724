// onchip.cuh -- the on-chip stable sort of up to 8192 rows by one warp or CTA.
#pragma once

#include "device_common.cuh"

namespace fmcs {
namespace {

// On-chip stable sort of one segment by a group of NT threads (one warp, or a
// CTA), IT rows per thread: one HBM read and one HBM write per row.
//
// Each row becomes a 64-bit compound: the key bits below the highest bit in
// which the segment's keys differ (the bits above are the same in every row),
// then the row's position in the segment.  Compounds are all distinct and
// compare like (key, position), so any order in which rows are bucketed gives
// the stable result.  (When both do not fit in 64 bits, the key's lowest `drop`
// bits stay beside it, by position, and decide between equal compounds.)
//   1. bucket = the compound's top ceil(log2 len) bits, about one row per
//      bucket for spread-out keys; rows take slots with shared-memory atomics;
//   2. an exclusive scan of the buckets; rows land bucketed, any order inside;
//   3. a row's place is its bucket's start plus the rows of the bucket with a
//      smaller compound; a row alone in its bucket is in its place.
// Few distinct keys spread as well, because the digit runs on into the position
// bits.  When some bucket holds more than kBucketRefine rows (skewed leading
// bits: one column's frequent code, followed by the next column), step 1 is
// refined: the rows of each bucket of 16 or more are spread over as many places
// by the 32 bits after the digit, interpolated between the lowest and highest
// that a sample of the bucket shows.  When some bucket even then holds more
// than kBucketMax rows, step 1 is done again: NT splitters, one compound taken
// somewhere in each NT-th of the segment and sorted across the group by a bitonic
// network, cut the rows into coarse buckets of about IT rows whatever the keys
// (binary search), and a coarse bucket of m rows is cut into m fine ones by
// interpolating between its two splitters.  Every step keeps the compounds' order.
// Should some bucket hold more than kBucketWorst rows after all (keys laid out
// against the sampled places), the whole segment is sorted by a network instead:
// step 3 is quadratic in a bucket's rows.
// The oids wait in shared memory in the order they were read; a compound's
// position bits find a row's oid when the segment is written out, so only
// compounds move.
//
// Bound: issue slots and shared-memory latency, about 230 instructions a row
// (the HBM traffic is 24 bytes a row for 8-byte keys).  A warp sorts a segment of
// up to 256 rows by itself: no block barriers, and three to four times as many
// rows in flight per SM as one small CTA per segment.  (One warp for 512 rows
// as well, 16 rows a lane, takes twice as long for one segment, 12.6 us
// against 7.0, which is what counts when there are few.)
// Measured against warp-level LSD passes up to 128 rows and LSD passes as the
// answer to skew: the tiers up to 512 rows of 384 instances of 64-bit keys
// (38.6M rows) 1,978 us before, 670 now; one 8192-row segment of Zipf codes 72
// before, 54 now.
// kBucketMax: 64 (a 67M-row Zipf plan takes 3.72 ms with 48 to 192, 4.00 with
// 16; 90,001 rows of it 241 us with 48 to 96 and 286 with 192, where a bucket is
// counted through for too long before the splitters take over).
constexpr uint32_t kBucketMax = 64;
// kBucketRefine: 24 (16 and 40 differ by 1 to 2%, either way by case; without the
// step the 90,001 rows take 198 us instead of 175).
constexpr uint32_t kBucketRefine = 24;
// kBucketWorst: coarse buckets hold IT rows on average, at random places hardly
// ever ten times as many.
constexpr uint32_t kBucketWorst = 128;

constexpr int pow2_ceil(int x)
{
    int p = 1;
    while (p < x) p <<= 1;
    return p;
}

// (off is accessed by 16-byte vectors, and the warps of a CTA have an array of
// these: both alignments are stated, whatever the members before)
// What only skewed segments need lies where the compounds go: as long as they are
// bucketed anew the rows' compounds are in registers.  Shared memory that is not
// used is L1, which holds the sectors in flight of a later round's random key
// reads: with these arrays beside cs a round of 16M rows in random order took 515
// us in segments of 2048 rows and 703 in segments of 2200, with them in it 454 and
// 502.
template <typename K, int NT, int IT>
struct alignas(16) OnchipSmem {
    static constexpr int kRows = NT * IT;
    static constexpr int kBins = pow2_ceil(kRows) < 128 ? 128 : pow2_ceil(kRows);
    struct Ranges {
        uint32_t lowest[kRows / 16 + 1], highest[kRows / 16 + 1];   // per large bucket (its start / 16): its sampled range
    };
    struct Splitters {
        unsigned long long spl[NT];   // sorted splitters
        uint32_t cst[NT];             // per coarse bucket: its start
        float cinv[NT];               // and its rows per unit of compound
    };
    union {
        unsigned long long cs[kRows];   // compounds, bucketed
        Ranges rg;
        Splitters sp;
    };
    uint32_t vals[kRows];           // oids by position
    alignas(16) uint32_t off[kBins + 4];   // per bucket: count -> start; then len
    unsigned long long any[NT / 32], all[NT / 32];   // per warp: OR and AND of its keys
    uint16_t lo[sizeof(K) == 8 ? kRows : 8];         // the keys' dropped low bits by position
    uint32_t tmp[NT / 32 + 1];
    uint32_t maxb;
};

// Exclusive scan of off[0, nb) by the block (nb a power of two, at most
// NT * IT, so at most 16 * NT), also leaving the largest count in *maxb.
// Thread t scans its own run of PER = nb / NT consecutive bins (one bin each
// for the first nb threads when nb < NT), read as vectors and summed, then,
// after the runs' totals are scanned across the block, read again and written
// back as exclusive offsets (the run is not held in registers across the
// barriers).  A run of NV > 1 16-byte vectors is visited starting at vector
// (t * PER / 32) mod NV, so that the 8 threads of a shared-memory wavefront
// touch 8 different bank groups instead of 2 to 4.
template <int NT, int PER>
__device__ __forceinline__ void scan_bin_runs(uint32_t *off, uint32_t nb, uint32_t *tmp, uint32_t *maxb)
{
    constexpr int NW = NT / 32;
    constexpr int VW = PER >= 4 ? 4 : PER;   // words per vector access
    constexpr int NV = PER / VW;             // vectors per run
    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const uint32_t b0 = threadIdx.x * PER;
    const bool mine = b0 < nb;
    const uint32_t rot = NV > 1 ? (threadIdx.x * PER / 32) : 0u;
    auto vec_of = [&](int q) -> uint32_t { return ((uint32_t)q + rot) & (uint32_t)(NV - 1); };
    auto ld = [&](uint32_t v, uint32_t (&x)[VW]) {
        if constexpr (VW == 4) {
            const uint4 w = reinterpret_cast<const uint4 *>(off + b0)[v];
            x[0] = w.x; x[1] = w.y; x[2] = w.z; x[3] = w.w;
        } else if constexpr (VW == 2) {
            const uint2 w = reinterpret_cast<const uint2 *>(off + b0)[v];
            x[0] = w.x; x[1] = w.y;
        } else {
            x[0] = off[b0 + v];
        }
    };
    uint32_t sum = 0, mx = 0;
    if (mine) {
#pragma unroll
        for (int q = 0; q < NV; ++q) {
            uint32_t x[VW];
            ld(vec_of(q), x);
#pragma unroll
            for (int i = 0; i < VW; ++i) {
                sum += x[i];
                mx = max(mx, x[i]);
            }
        }
    }
    uint32_t incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, incl, o);
        if (lane >= o) incl += y;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mx = max(mx, __shfl_xor_sync(0xFFFFFFFFu, mx, o));
    if (lane == 31) tmp[warp] = incl;
    if (lane == 0 && mx) atomicMax(maxb, mx);
    __syncthreads();
    if (warp == 0) {
        const uint32_t w = lane < NW ? tmp[lane] : 0u;
        uint32_t wi = w;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, wi, o);
            if (lane >= o) wi += y;
        }
        if (lane < NW) tmp[lane] = wi - w;
    }
    __syncthreads();
    if (mine) {
        const uint32_t run = tmp[warp] + incl - sum;
        // the run's vectors in visiting order, with their sums
        uint32_t x[NV][VW], vs[NV];
#pragma unroll
        for (int q = 0; q < NV; ++q) {
            ld(vec_of(q), x[q]);
            vs[q] = 0;
#pragma unroll
            for (int i = 0; i < VW; ++i) vs[q] += x[q][i];
        }
#pragma unroll
        for (int q = 0; q < NV; ++q) {
            // the vector's first offset: the run's plus every vector before it
            uint32_t r = run;
#pragma unroll
            for (int u = 0; u < NV; ++u) r += vec_of(u) < vec_of(q) ? vs[u] : 0u;
#pragma unroll
            for (int i = 0; i < VW; ++i) {
                const uint32_t c = x[q][i];
                x[q][i] = r;
                r += c;
            }
            const uint32_t v = vec_of(q);
            if constexpr (VW == 4) reinterpret_cast<uint4 *>(off + b0)[v] = make_uint4(x[q][0], x[q][1], x[q][2], x[q][3]);
            else if constexpr (VW == 2) reinterpret_cast<uint2 *>(off + b0)[v] = make_uint2(x[q][0], x[q][1]);
            else off[b0 + v] = x[q][0];
        }
    }
    __syncthreads();
}

template <int NT>
__device__ __forceinline__ void block_scan_bins(uint32_t *off, uint32_t nb, uint32_t *tmp, uint32_t *maxb)
{
    switch (nb >= (uint32_t)NT ? nb / NT : 1u) {
    case 1: scan_bin_runs<NT, 1>(off, nb, tmp, maxb); break;
    case 2: scan_bin_runs<NT, 2>(off, nb, tmp, maxb); break;
    case 4: scan_bin_runs<NT, 4>(off, nb, tmp, maxb); break;
    case 8: scan_bin_runs<NT, 8>(off, nb, tmp, maxb); break;
    default: scan_bin_runs<NT, 16>(off, nb, tmp, maxb); break;
    }
}

// Exclusive scan of off[0, nb) by one warp, 128 bins a step (bins past nb are
// zero: off holds at least 128).  Returns the largest count.
__device__ __forceinline__ uint32_t warp_scan_bins(uint32_t *off, uint32_t nb)
{
    const uint32_t lane = lane_id();
    uint32_t carry = 0, mx = 0;
    for (uint32_t q = 0; q < nb; q += 128) {
        uint4 w = reinterpret_cast<const uint4 *>(off + q)[lane];
        mx = max(mx, max(max(w.x, w.y), max(w.z, w.w)));
        const uint32_t sum = w.x + w.y + w.z + w.w;
        uint32_t incl = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, incl, o);
            if ((int)lane >= o) incl += y;
        }
        uint32_t r = carry + incl - sum;
        carry += __shfl_sync(0xFFFFFFFFu, incl, 31);
        uint32_t t;
        t = w.x; w.x = r; r += t;
        t = w.y; w.y = r; r += t;
        t = w.z; w.z = r; r += t;
        w.w = r;
        reinterpret_cast<uint4 *>(off + q)[lane] = w;
    }
    return __reduce_max_sync(0xFFFFFFFFu, mx);
}

template <int NT>
__device__ __forceinline__ void group_sync()
{
    if constexpr (NT == 32) __syncwarp();
    else __syncthreads();
}

// off[0, nb) scanned by the group, off[nb] = len; returns the largest count.
// Synchronizes the group before and after.
template <typename K, int NT, int IT>
__device__ __forceinline__ uint32_t group_scan_bins(OnchipSmem<K, NT, IT> &sm, uint32_t nb, uint32_t len)
{
    group_sync<NT>();
    const uint32_t tid = NT == 32 ? lane_id() : threadIdx.x;
    uint32_t mx;
    if constexpr (NT == 32) {
        mx = warp_scan_bins(sm.off, nb);
        if (tid == 0) sm.off[nb] = len;
    } else {
        if (tid == 0) sm.off[nb] = len;
        block_scan_bins<NT>(sm.off, nb, sm.tmp, &sm.maxb);
        mx = sm.maxb;
    }
    group_sync<NT>();
    return mx;
}

template <int NT>
__device__ __forceinline__ void zero_bins(uint32_t *off, uint32_t nb, uint32_t tid)
{
    // whole vectors; nb is a power of two >= 32
    for (uint32_t i = tid; i < nb / 4; i += NT) reinterpret_cast<uint4 *>(off)[i] = make_uint4(0, 0, 0, 0);
}

// Order of two compounds: by value, except that compounds whose key bits are
// equal are decided by the dropped low bits first (drop > 0), then by position.
template <typename K, int NT, int IT>
__device__ __forceinline__ bool comp_less(const OnchipSmem<K, NT, IT> &sm, unsigned long long x, unsigned long long y,
                                          uint32_t drop, uint32_t nbits)
{
    bool less = x < y;
    if constexpr (sizeof(K) == 8) {
        const uint32_t pmask = (1u << nbits) - 1u;
        if (drop && (x ^ y) <= pmask) {
            const uint32_t lx = sm.lo[(uint32_t)x & pmask], ly = sm.lo[(uint32_t)y & pmask];
            less = lx < ly || (lx == ly && less);
        }
    }
    return less;
}

// Where splitter t of len rows is taken: somewhere in the t-th of NT equal parts.
// (The parts' beginnings are an even stride apart.  Rows whose keys repeat with a
// period that shares a factor with it, as in joined or generated tables, would
// show a few of their keys only, and the rows of all others would share a bucket:
// a round over 296 segments of 8192 rows, codes i % 8 and one far key each, 3.35
// ms with places at the beginnings and 0.18 with these; 64-bit keys of a few low
// bits and one highest 18.8 and 0.32.)
template <int NT>
__device__ __forceinline__ uint32_t splitter_place(uint32_t t, uint32_t len)
{
    const uint32_t a = t * len / NT, z = (t + 1) * len / NT;   // (len <= 2^13)
    uint32_t h = (t + 1) * 0x9E3779B9u;   // mixed: an odd constant, a fold, another
    h = (h ^ (h >> 15)) * 0x2C1B3C6Du;
    return a + __umulhi(h, z - a);
}

// The dropped low bits and the position of a compound, as one word.
template <typename K, int NT, int IT>
__device__ __forceinline__ uint32_t low_word(const OnchipSmem<K, NT, IT> &sm, unsigned long long x, uint32_t nbits)
{
    const uint32_t p = (uint32_t)x & ((1u << nbits) - 1u);
    return ((uint32_t)sm.lo[p] << nbits) | p;
}

// Rows of the bucket [bs, bs + bn) that sort before x, when the keys' low bits are
// dropped from the compounds.  As long as no other row with the same kept bits is
// met (spread-out keys: hardly ever), the compounds decide; then the count starts
// again and looks at the dropped bits of such rows.  (A round over 16M rows of
// 64-bit keys in segments of 2048: 405 us when every comparison looked at them, 336
// so; 2.4M rows of 200 values in segments of 2000 186 us and 144.  Out of line, as
// its registers and instructions weigh on the segments that drop nothing: the first
// radix round of 16M 50-bit keys 557 us with it inline, 544 without.)
template <typename K, int NT, int IT>
__device__ __noinline__ uint32_t rank_dropped(const OnchipSmem<K, NT, IT> &sm, uint32_t bs, uint32_t bn,
                                              unsigned long long x, uint32_t nbits)
{
    const uint32_t pmask = (1u << nbits) - 1u;
    uint32_t r = 0, same = 0;
    for (uint32_t q = 0; q < bn && same < 2u; ++q) {
        const unsigned long long y = sm.cs[bs + q];
        r += y < x;
        same += (y ^ x) <= pmask;
    }
    if (same > 1u) {
        const uint32_t xl = low_word(sm, x, nbits);
        r = 0;
        for (uint32_t q = 0; q < bn; ++q) {
            const unsigned long long y = sm.cs[bs + q];
            r += (y ^ x) <= pmask ? low_word(sm, y, nbits) < xl : y < x;
        }
    }
    return r;
}

// The fine bucket of x among the m rows of coarse bucket bi, when the keys' low
// bits are dropped: by the kept bits (inv rows per unit of compound), or, where
// they are the same in both its splitters, by dropped bits and position.
// (Otherwise the rows of a key that is frequent enough to be many splitters would
// share a fine bucket: a round over 2.4M 64-bit keys of 16 values in segments of
// 8000 rows 449 us, 285 so.)  Out of line, as rank_dropped is.
template <typename K, int NT, int IT>
__device__ __noinline__ uint32_t fine_dropped(const OnchipSmem<K, NT, IT> &sm, uint32_t bi, uint32_t m, float inv,
                                              unsigned long long x, uint32_t nbits)
{
    const uint32_t pmask = (1u << nbits) - 1u;
    const unsigned long long a = bi ? sm.sp.spl[bi] : 0ull;
    if (bi && bi + 1 < (uint32_t)NT) {
        const unsigned long long z = sm.sp.spl[bi + 1];
        if ((a ^ z) <= pmask) {
            const uint32_t al = low_word(sm, a, nbits);
            const float span = (float)(low_word(sm, z, nbits) - al) + 1.0f;
            return min((uint32_t)((float)(low_word(sm, x, nbits) - al) * __fdividef((float)m, span)), m - 1u);
        }
    }
    const unsigned long long kept = ~(unsigned long long)pmask;
    return min((uint32_t)(__ull2float_rn((x & kept) - (a & kept)) * inv), m - 1u);
}

// The splitters of step 1's second try: NT compounds of the segment (in sm.cs
// by position), sorted into sm.sp.spl, which takes sm.cs's place.  Out of line: it runs for skewed segments
// only, and its registers must not weigh on the others.
template <typename K, int NT, int IT>
__device__ __noinline__ void sort_splitters(OnchipSmem<K, NT, IT> &sm, uint32_t len, uint32_t drop, uint32_t nbits)
{
    const uint32_t tid = NT == 32 ? lane_id() : threadIdx.x;
    unsigned long long x = sm.cs[splitter_place<NT>(tid, len)];
    group_sync<NT>();   // the splitters go where the compounds were
#pragma unroll 1
    for (uint32_t k = 2; k <= (uint32_t)NT; k <<= 1) {
#pragma unroll 1
        for (uint32_t j = k >> 1; j > 0; j >>= 1) {
            unsigned long long y;
            if (j < 32) {
                y = __shfl_xor_sync(0xFFFFFFFFu, x, j);
            } else {
                sm.sp.spl[tid] = x;
                group_sync<NT>();
                y = sm.sp.spl[tid ^ j];
                group_sync<NT>();
            }
            const bool lower = ((tid & k) == 0) == ((tid & j) == 0);
            x = comp_less(sm, y, x, drop, nbits) == lower ? y : x;
        }
    }
    sm.sp.spl[tid] = x;
}

// The compounds in sm.cs sorted in place, len of them, 2^nbits >= len: a bitonic
// network whose comparisons all point upwards (each merge starts by comparing
// mirrored places), so that the places past len need not exist.  91 steps for
// 8192 rows whatever the keys; it runs for keys that defeat the splitters only.
template <typename K, int NT, int IT>
__device__ __noinline__ void sort_network(OnchipSmem<K, NT, IT> &sm, uint32_t len, uint32_t drop, uint32_t nbits)
{
    const uint32_t tid = NT == 32 ? lane_id() : threadIdx.x;
    const uint32_t half = 1u << (nbits - 1u);
#pragma unroll 1
    for (uint32_t k = 2; k <= 2u * half; k <<= 1) {
#pragma unroll 1
        for (uint32_t h = k >> 1; h > 0; h >>= 1) {
            group_sync<NT>();
#pragma unroll 1
            for (uint32_t t = tid; t < half; t += NT) {
                const uint32_t i = 2u * t - (t & (h - 1u));   // bit h of the place is 0
                const uint32_t j = h == k >> 1 ? i ^ (k - 1u) : i + h;
                if (j < len) {
                    const unsigned long long x = sm.cs[i], y = sm.cs[j];
                    if (comp_less(sm, y, x, drop, nbits)) {
                        sm.cs[i] = y;
                        sm.cs[j] = x;
                    }
                }
            }
        }
    }
    group_sync<NT>();
}

// The compounds' layout, for reading sm.cs back.
struct OnchipInfo {
    unsigned long long prefix;   // the key bits every row shares
    uint32_t nbits, drop;
    bool same;                   // every key is the same: nothing was sorted, sm.cs is not written
};

// Key and position of a sorted compound.
template <typename K, int NT, int IT>
__device__ __forceinline__ unsigned long long onchip_key(const OnchipSmem<K, NT, IT> &sm, const OnchipInfo &f,
                                                         unsigned long long x, uint32_t *pos)
{
    const uint32_t q = (uint32_t)x & ((1u << f.nbits) - 1u);
    unsigned long long k = f.prefix | ((x >> f.nbits) << f.drop);
    if constexpr (sizeof(K) == 8) {
        if (f.drop) k |= sm.lo[q];
    }
    *pos = q;
    return k;
}

// Sorts the keys c[j] (row wbase + j * 32 + lane of len, j < steps) into sm.cs.
// sm.vals is the caller's (the oids by position).  The group is synchronized
// on return, after which sm.cs, sm.vals and sm.lo may be read.
template <typename K, int NT, int IT>
__device__ __forceinline__ OnchipInfo onchip_core(OnchipSmem<K, NT, IT> &sm, unsigned long long (&c)[IT],
                                                  uint32_t steps, uint32_t wbase, uint32_t len)
{
    constexpr int NW = NT / 32;
    const uint32_t lane = lane_id();
    const uint32_t warp = NT == 32 ? 0u : threadIdx.x >> 5;
    const uint32_t tid = NT == 32 ? lane : threadIdx.x;
    const uint32_t nbits = max(5u, 32u - (uint32_t)__clz(len - 1u));   // ceil(log2(len)), at least a vector of bins
    const uint32_t nb = 1u << nbits;
    zero_bins<NT>(sm.off, NT == 32 && nb < 128 ? 128u : nb, tid);
    if (tid == 0) sm.maxb = 0;
    unsigned long long any = 0ull, all = ~0ull;
#pragma unroll
    for (int j = 0; j < IT; ++j) {
        const uint32_t p = wbase + j * 32 + lane;
        if (j < (int)steps && p < len) {
            any |= c[j];
            all &= c[j];
        }
    }
    if constexpr (sizeof(K) == 8) {
        any = ((unsigned long long)__reduce_or_sync(0xFFFFFFFFu, (uint32_t)(any >> 32)) << 32) |
              __reduce_or_sync(0xFFFFFFFFu, (uint32_t)any);
        all = ((unsigned long long)__reduce_and_sync(0xFFFFFFFFu, (uint32_t)(all >> 32)) << 32) |
              __reduce_and_sync(0xFFFFFFFFu, (uint32_t)all);
    } else {
        any = __reduce_or_sync(0xFFFFFFFFu, (uint32_t)any);
        all = __reduce_and_sync(0xFFFFFFFFu, (uint32_t)all);
    }
    if constexpr (NT > 32) {
        if (lane == 0) {
            sm.any[warp] = any;
            sm.all[warp] = all;
        }
    }
    group_sync<NT>();
    if constexpr (NT > 32) {
        any = 0ull;
        all = ~0ull;
#pragma unroll
        for (int w = 0; w < NW; ++w) {
            any |= sm.any[w];
            all &= sm.all[w];
        }
    }
    const unsigned long long diff = any & ~all;
    if (diff == 0ull) return OnchipInfo{all, nbits, 0u, true};
    const uint32_t top = 64u - (uint32_t)__clzll((long long)diff);   // bits [0, top) differ somewhere
    const unsigned long long low = top >= 64u ? ~0ull : ((1ull << top) - 1ull);
    const unsigned long long prefix = all & ~low;                    // the bits every row shares
    // (only 8-byte keys reach past 64 bits: a segment has at most 2^13 rows)
    const uint32_t drop = sizeof(K) == 8 && top + nbits > 64u ? top + nbits - 64u : 0u;
    uint32_t shift = top - drop;   // bucket = compound >> shift: its top nbits
    const uint32_t pmask = nb - 1u;
    uint32_t bk[IT];   // bucket << 16 | slot, then bucket start | size << 16
#pragma unroll
    for (int j = 0; j < IT; ++j) {
        const uint32_t p = wbase + j * 32 + lane;
        if (j < (int)steps && p < len) {
            if constexpr (sizeof(K) == 8) {
                if (drop) sm.lo[p] = (uint16_t)(c[j] & ((1ull << drop) - 1ull));
            }
            c[j] = (((c[j] & low) >> drop) << nbits) | p;
            const uint32_t bi = (uint32_t)(c[j] >> shift);
            bk[j] = (bi << 16) | atomicAdd(&sm.off[bi], 1u);
        }
    }
    uint32_t maxb = group_scan_bins<K, NT, IT>(sm, nb, len);   // (uniform across the group)
    if (maxb > kBucketRefine) {
        // large buckets: cut by the 32 bits after the digit, interpolated between
        // the lowest and the highest that one row a thread shows
        for (uint32_t i = tid; i <= len / 16; i += NT) {
            sm.rg.lowest[i] = 0xFFFFFFFFu;
            sm.rg.highest[i] = 0u;
        }
        if (tid == 0) sm.maxb = 0;
        group_sync<NT>();
        auto next32 = [&](unsigned long long x) -> uint32_t {
            return shift >= 32u ? (uint32_t)(x >> (shift - 32u)) : (uint32_t)(x << (32u - shift));
        };
#pragma unroll
        for (int j = 0; j < IT; ++j) {
            const uint32_t p = wbase + j * 32 + lane;
            if (j < (int)steps && p < len) {
                const uint32_t bi = bk[j] >> 16;
                const uint32_t bs = sm.off[bi], m = sm.off[bi + 1] - bs;
                bk[j] = bs | (m << 16);
                if (j == 0 && m >= 16u) {
                    const uint32_t d = next32(c[j]);
                    atomicMin(&sm.rg.lowest[bs >> 4], d);
                    atomicMax(&sm.rg.highest[bs >> 4], d);
                }
            }
        }
        group_sync<NT>();
        zero_bins<NT>(sm.off, NT == 32 && nb < 128 ? 128u : nb, tid);
        group_sync<NT>();
#pragma unroll
        for (int j = 0; j < IT; ++j) {
            const uint32_t p = wbase + j * 32 + lane;
            if (j < (int)steps && p < len) {
                uint32_t fb = bk[j] & 0xFFFFu;
                const uint32_t m = bk[j] >> 16;
                if (m >= 16u) {
                    const uint32_t a = sm.rg.lowest[fb >> 4], z = sm.rg.highest[fb >> 4], d = next32(c[j]);
                    // (no row sampled: a > z, everything goes to the first)
                    if (d > a && z > a) {
                        const float f = (float)(d - a) * __fdividef((float)m, (float)(z - a));
                        fb += min((uint32_t)f, m - 1u);
                    }
                }
                bk[j] = (fb << 16) | atomicAdd(&sm.off[fb], 1u);
            }
        }
        maxb = group_scan_bins<K, NT, IT>(sm, nb, len);
    }
    if (maxb > kBucketMax) {
        // skewed: bucket by splitters (uniform across the group)
#pragma unroll
        for (int j = 0; j < IT; ++j) {
            const uint32_t p = wbase + j * 32 + lane;
            if (j < (int)steps && p < len) sm.cs[p] = c[j];
        }
        zero_bins<NT>(sm.off, NT == 32 ? 128u : (uint32_t)NT, tid);
        if (tid == 0) sm.maxb = 0;
        group_sync<NT>();
        sort_splitters<K, NT, IT>(sm, len, drop, nbits);
        group_sync<NT>();
#pragma unroll
        for (int j = 0; j < IT; ++j) {
            const uint32_t p = wbase + j * 32 + lane;
            if (j < (int)steps && p < len) {
                // the last splitter not above the row (bucket 0 for all below splitter 1)
                uint32_t bi = 0;
#pragma unroll 1
                for (uint32_t h = NT / 2; h > 0; h >>= 1)
                    if (!comp_less(sm, c[j], sm.sp.spl[bi + h], drop, nbits)) bi += h;
                bk[j] = bi;
                atomicAdd(&sm.off[bi], 1u);
            }
        }
        group_scan_bins<K, NT, IT>(sm, NT, len);
        // (with dropped bits the position is not next in the order: the
        // interpolation leaves it out)
        const unsigned long long cmask = drop ? ~(unsigned long long)pmask : ~0ull;
        {
            const unsigned long long a = tid ? sm.sp.spl[tid] & cmask : 0ull;
            const unsigned long long z = tid + 1 < (uint32_t)NT ? sm.sp.spl[tid + 1] & cmask
                                                                : ~0ull >> (64u - (top - drop) - nbits);
            const uint32_t s0 = sm.off[tid];
            sm.sp.cst[tid] = s0;
            sm.sp.cinv[tid] = (float)(sm.off[tid + 1] - s0) / ((float)(z - a) + 1.0f);
        }
        group_sync<NT>();
        zero_bins<NT>(sm.off, NT == 32 && nb < 128 ? 128u : nb, tid);
        if (tid == 0) sm.maxb = 0;
        group_sync<NT>();
#pragma unroll
        for (int j = 0; j < IT; ++j) {
            const uint32_t p = wbase + j * 32 + lane;
            if (j < (int)steps && p < len) {
                const uint32_t bi = bk[j];
                const uint32_t s0 = sm.sp.cst[bi];
                const uint32_t e0 = bi + 1 < (uint32_t)NT ? sm.sp.cst[bi + 1] : len;
                uint32_t fb = s0;
                if (sizeof(K) == 8 && drop) {
                    fb += fine_dropped(sm, bi, e0 - s0, sm.sp.cinv[bi], c[j], nbits);
                } else {
                    const unsigned long long a = bi ? sm.sp.spl[bi] : 0ull;
                    fb += min((uint32_t)(__ull2float_rn(c[j] - a) * sm.sp.cinv[bi]), e0 - s0 - 1u);
                }
                bk[j] = (fb << 16) | atomicAdd(&sm.off[fb], 1u);
            }
        }
        if (group_scan_bins<K, NT, IT>(sm, nb, len) > kBucketWorst) {   // (uniform across the group)
#pragma unroll
            for (int j = 0; j < IT; ++j) {
                const uint32_t p = wbase + j * 32 + lane;
                if (j < (int)steps && p < len) sm.cs[p] = c[j];
            }
            sort_network<K, NT, IT>(sm, len, drop, nbits);
            return OnchipInfo{prefix, nbits, drop, false};
        }
    }
    // rows land bucketed; each keeps its bucket's start and size
#pragma unroll
    for (int j = 0; j < IT; ++j) {
        const uint32_t p = wbase + j * 32 + lane;
        if (j < (int)steps && p < len) {
            const uint32_t bi = bk[j] >> 16, slot = bk[j] & 0xFFFFu;
            const uint32_t bs = sm.off[bi], be = sm.off[bi + 1];
            sm.cs[bs + slot] = c[j];
            bk[j] = bs | ((be - bs) << 16);
        } else {
            bk[j] = 0;
        }
    }
    group_sync<NT>();
    // a row alone in its bucket is in its place; the others count the rows of
    // their bucket that sort before them
#pragma unroll
    for (int j = 0; j < IT; ++j) {
        const uint32_t bs = bk[j] & 0xFFFFu, bn = bk[j] >> 16;
        if (bn > 1) {
            uint32_t r = 0;
            if (sizeof(K) < 8 || drop == 0) {
                for (uint32_t q = 0; q < bn; ++q) r += sm.cs[bs + q] < c[j];
            } else {
                r = rank_dropped(sm, bs, bn, c[j], nbits);
            }
            bk[j] = (bs + r) | 0x80000000u;   // its place; it moves
        }
    }
    group_sync<NT>();
#pragma unroll
    for (int j = 0; j < IT; ++j)
        if (bk[j] >> 31) sm.cs[bk[j] & 0xFFFFu] = c[j];
    group_sync<NT>();
    return OnchipInfo{prefix, nbits, drop, false};
}

}  // namespace
}  // namespace fmcs
