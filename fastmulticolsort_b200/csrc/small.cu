// small.cu -- a whole sort plan, or one sort round, over at most kSmallRows rows
// in ONE launch of one CTA.
//
// At this size a plan's time is launches and the gaps between them (stitch,
// classification, a tier, three scan passes, copies back), not work.  The CTA
// keeps the rows on chip: it sorts by the plan's banks from the last to the
// first (every sort is stable, so the result is the reference's round by round
// order, src/composer.cpp:48-135), building each bank's keys from the columns as
// it goes, and a segmented round sorts by its bank and then by its segment.
// Group ids are an adjacent difference over the banks and one scan.
// Bound: latency, one SM's barriers and shared memory.  3,001 rows, one 50-bit
// bank: 10 us in this kernel, 26 us the call (41 by the general path's launches).
// The limit is what one CTA's shared memory holds.  There, at 8,192 rows, one
// launch against the general path: [50] 38 us (49), [17,33] 57 (83), [64,20] 82
// (100), six columns in [59,7] 84 (86); only three rounds driven one by one lose,
// 188 (180).
#include "device_common.cuh"
#include "fmcs_internal.h"
#include "onchip.cuh"

#include <algorithm>

namespace fmcs {
namespace {

constexpr int kSmallSlices = 32;
constexpr int kSmallBanks = 16;

struct SmallParams {
    StitchSlice s[kSmallSlices];
    uint8_t first[kSmallBanks + 1];   // bank b: slices [first[b], first[b + 1])
    uint32_t nbanks, n;
    const uint32_t *order_in;    // NULL: rows in row order
    const uint32_t *in_group;    // NULL: one segment
    uint32_t *order_out;         // may be order_in
    uint32_t *group_out;         // may be NULL
    void *keys_out;              // the first bank's keys in the final order, or NULL
    uint32_t key_bytes;
    uint32_t *d_ngroups;
};

__device__ __forceinline__ uint64_t load_code(const StitchSlice &s, uint32_t row)
{
    switch (s.src_bytes) {
    case 1: return ((const uint8_t *)s.src)[row];
    case 2: return ((const uint16_t *)s.src)[row];
    case 4: return ((const uint32_t *)s.src)[row];
    default: return ((const uint64_t *)s.src)[row];
    }
}

// Keys of bank b of the rows row[j].
template <int IT>
__device__ __forceinline__ void bank_keys(const SmallParams &p, uint32_t b, const uint32_t (&row)[IT], uint32_t valid,
                                          unsigned long long (&key)[IT])
{
#pragma unroll
    for (int j = 0; j < IT; ++j) key[j] = 0ull;
    for (int i = p.first[b]; i < p.first[b + 1]; ++i) {
        const StitchSlice sl = p.s[i];
        const uint64_t mask = sl.width >= 64 ? ~0ull : ((1ull << sl.width) - 1);
        const uint64_t flip = sl.invert ? mask : 0ull;
        uint64_t v[IT];
#pragma unroll
        for (int j = 0; j < IT; ++j) v[j] = (valid >> j) & 1u ? load_code(sl, row[j]) : 0ull;
#pragma unroll
        for (int j = 0; j < IT; ++j) {
            const uint64_t x = ((v[j] >> sl.rshift) & mask) ^ flip;
            key[j] = sl.width >= 64 ? x : ((key[j] << sl.width) | x);
        }
    }
}

template <int NT, int IT>
struct alignas(16) SmallSmem {
    OnchipSmem<uint64_t, NT, IT> sort;
    uint16_t run[NT * IT];      // segment of each input position
    uint32_t wsum[NT / 32];
};

// Inclusive count of the flags (bit j: row wbase + j * 32 + lane) up to each row,
// and the total.
template <int NT, int IT>
__device__ __forceinline__ uint32_t count_flags(uint32_t *wsum, uint32_t flags, uint32_t (&incl)[IT])
{
    const uint32_t lane = lane_id(), warp = threadIdx.x >> 5;
    uint32_t sum = 0;
#pragma unroll
    for (int j = 0; j < IT; ++j) {
        const uint32_t bal = __ballot_sync(0xFFFFFFFFu, (flags >> j) & 1u);
        incl[j] = sum + __popc(bal & (lanemask_lt() | (1u << lane)));
        sum += __popc(bal);
    }
    if (lane == 0) wsum[warp] = sum;
    __syncthreads();
    const uint32_t w = lane < (uint32_t)(NT / 32) ? wsum[lane] : 0u;
    const uint32_t before = __reduce_add_sync(0xFFFFFFFFu, lane < warp ? w : 0u);
    const uint32_t total = __reduce_add_sync(0xFFFFFFFFu, w);
#pragma unroll
    for (int j = 0; j < IT; ++j) incl[j] += before;
    __syncthreads();
    return total;
}

template <int NT, int IT>
__global__ void __launch_bounds__(NT, 1) small_plan_kernel(const __grid_constant__ SmallParams p)
{
    kernel_prologue();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    SmallSmem<NT, IT> &sm = *reinterpret_cast<SmallSmem<NT, IT> *>(smem_raw);
    const uint32_t n = p.n, lane = lane_id(), warp = threadIdx.x >> 5;
    const uint32_t steps = (n + NT - 1) / NT;
    const uint32_t wbase = warp * steps * 32;
    uint32_t valid = 0;   // bit j: this thread has a row j
    uint32_t pos[IT];     // the input position of the row now at wbase + j * 32 + lane
#pragma unroll
    for (int j = 0; j < IT; ++j) {
        const uint32_t i = wbase + j * 32 + lane;
        pos[j] = i;
        if (j < (int)steps && i < n) valid |= 1u << j;
    }
    if (p.in_group) {
        uint32_t flags = 0, run[IT];
#pragma unroll
        for (int j = 0; j < IT; ++j)
            if ((valid >> j) & 1u && (pos[j] == 0 || p.in_group[pos[j]] != p.in_group[pos[j] - 1])) flags |= 1u << j;
        count_flags<NT, IT>(sm.wsum, flags, run);
#pragma unroll
        for (int j = 0; j < IT; ++j)
            if ((valid >> j) & 1u) sm.run[pos[j]] = (uint16_t)(run[j] - 1u);
        __syncthreads();
    }
    auto rows_of = [&](uint32_t (&row)[IT]) {
#pragma unroll
        for (int j = 0; j < IT; ++j) row[j] = p.order_in && (valid >> j) & 1u ? p.order_in[pos[j]] : pos[j];
    };
    // sorts, last bank first, then by segment; key[] ends as the keys of the
    // last sort in its order
    const uint32_t nsorts = p.nbanks + (p.in_group ? 1u : 0u);
    unsigned long long key[IT];
    for (uint32_t k = 0; k < nsorts; ++k) {
        const bool by_run = k == p.nbanks;
        if (by_run) {
#pragma unroll
            for (int j = 0; j < IT; ++j) key[j] = (valid >> j) & 1u ? sm.run[pos[j]] : 0u;
        } else {
            uint32_t row[IT];
            rows_of(row);
            bank_keys<IT>(p, p.nbanks - 1 - k, row, valid, key);
        }
#pragma unroll
        for (int j = 0; j < IT; ++j)
            if ((valid >> j) & 1u) sm.sort.vals[wbase + j * 32 + lane] = pos[j];
        const OnchipInfo f = onchip_core<uint64_t, NT, IT>(sm.sort, key, steps, wbase, n);
        if (f.same) {   // (key[] still holds the keys)
            __syncthreads();
            continue;
        }
#pragma unroll
        for (int j = 0; j < IT; ++j) {
            if ((valid >> j) & 1u) {
                uint32_t q;
                key[j] = onchip_key(sm.sort, f, sm.sort.cs[wbase + j * 32 + lane], &q);
                pos[j] = sm.sort.vals[q];
            }
        }
        __syncthreads();
    }
    uint32_t row[IT];
    rows_of(row);   // every read of order_in comes before the barriers below, its writes after
    const bool have = nsorts == 1;   // key[] is the only bank's
    if (p.keys_out && !have) bank_keys<IT>(p, 0, row, valid, key);
    if (p.keys_out) {
#pragma unroll
        for (int j = 0; j < IT; ++j) {
            if ((valid >> j) & 1u) {
                const uint32_t i = wbase + j * 32 + lane;
                if (p.key_bytes == 2) ((uint16_t *)p.keys_out)[i] = (uint16_t)key[j];
                else if (p.key_bytes == 4) ((uint32_t *)p.keys_out)[i] = (uint32_t)key[j];
                else ((uint64_t *)p.keys_out)[i] = key[j];
            }
        }
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < IT; ++j)
        if ((valid >> j) & 1u) p.order_out[wbase + j * 32 + lane] = row[j];
    if (!p.group_out && !p.d_ngroups) return;
    // a group starts where a bank's key or the segment differs from the row before
    uint32_t flags = 0;
    for (uint32_t k = 0; k < nsorts; ++k) {
        if (!have) {
            if (k == p.nbanks) {
#pragma unroll
                for (int j = 0; j < IT; ++j) key[j] = (valid >> j) & 1u ? sm.run[pos[j]] : 0u;
            } else {
                bank_keys<IT>(p, k, row, valid, key);
            }
        }
#pragma unroll
        for (int j = 0; j < IT; ++j)
            if ((valid >> j) & 1u) sm.sort.cs[wbase + j * 32 + lane] = key[j];
        __syncthreads();
#pragma unroll
        for (int j = 0; j < IT; ++j) {
            const uint32_t i = wbase + j * 32 + lane;
            if ((valid >> j) & 1u && (i == 0 || sm.sort.cs[i - 1] != key[j])) flags |= 1u << j;
        }
        __syncthreads();
    }
    uint32_t incl[IT];
    const uint32_t total = count_flags<NT, IT>(sm.wsum, flags, incl);
    if (p.group_out) {
#pragma unroll
        for (int j = 0; j < IT; ++j)
            if ((valid >> j) & 1u) p.group_out[wbase + j * 32 + lane] = incl[j] - 1u;
    }
    if (p.d_ngroups && threadIdx.x == 0) *p.d_ngroups = total;
}

template <int NT, int IT>
int launch_small_t(fmcs_ctx *ctx, const SmallParams &p, const char *name)
{
    const size_t smem = sizeof(SmallSmem<NT, IT>);
    const int rc = raise_smem(ctx, (const void *)small_plan_kernel<NT, IT>, smem);
    if (rc) return rc;
    LaunchScope ls_(ctx, name);
    const cudaError_t e = launch_k(small_plan_kernel<NT, IT>, 1, NT, smem, ctx->stream, p);
    return e == cudaSuccess ? FMCS_OK : cuda_fail(ctx, e, "small plan launch");
}

int launch_small(fmcs_ctx *ctx, const SmallParams &p, bool plan)
{
    // as few rows a thread as the block allows: the steps are a serial chain
    // (profiled as a plan by its own name; as a round under the name of the
    // on-chip tier of that capacity, the one sort of a segment that it is)
    return p.n <= 1024   ? launch_small_t<256, 4>(ctx, p, plan ? "small_plan" : "block_sort_1024")
           : p.n <= 4096 ? launch_small_t<1024, 4>(ctx, p, plan ? "small_plan" : "block_sort_4096")
                         : launch_small_t<1024, 8>(ctx, p, plan ? "small_plan" : "block_sort_8192");
}

}  // namespace

bool small_plan_fits(uint64_t n, const int *nslices, uint32_t nbanks)
{
    if (n > kSmallRows || nbanks > (uint32_t)kSmallBanks) return false;
    int total = 0;
    for (uint32_t b = 0; b < nbanks; ++b) total += nslices[b];
    return total <= kSmallSlices;
}

int launch_small_plan(fmcs_ctx *ctx, const StitchSlice *slices, const int *nslices, uint32_t nbanks, uint64_t n,
                      uint32_t *order_out, uint32_t *group_out, uint32_t *d_ngroups)
{
    SmallParams p{};
    int at = 0;
    for (uint32_t b = 0; b < nbanks; ++b) {
        p.first[b] = (uint8_t)at;
        for (int k = 0; k < nslices[b]; ++k, ++at) p.s[at] = slices[at];
    }
    p.first[nbanks] = (uint8_t)at;
    p.nbanks = nbanks;
    p.n = (uint32_t)n;
    p.order_out = order_out;
    p.group_out = group_out;
    p.d_ngroups = d_ngroups;
    return launch_small(ctx, p, true);
}

int launch_small_round(fmcs_ctx *ctx, const void *bank, uint32_t bank_bytes, uint32_t key_bits, const uint32_t *order_in,
                       const uint32_t *in_group, uint32_t *order_out, uint32_t *group_out, void *keys_out, uint64_t n,
                       uint32_t *d_ngroups)
{
    SmallParams p{};
    p.s[0] = StitchSlice{bank, bank_bytes, 0u, key_bits, 0u};
    p.first[1] = 1;
    p.nbanks = 1;
    p.n = (uint32_t)n;
    p.order_in = order_in;
    p.in_group = in_group;
    p.order_out = order_out;
    p.group_out = group_out;
    p.keys_out = keys_out;
    p.key_bytes = bank_bytes;
    p.d_ngroups = group_out ? d_ngroups : nullptr;
    return launch_small(ctx, p, false);
}

}  // namespace fmcs
