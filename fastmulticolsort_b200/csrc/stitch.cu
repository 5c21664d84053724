// stitch.cu -- (a) bit stitching of one bank in ONE pass.
//
// The reference builds a bank slice by slice with whole-column AVX2 passes:
// ShiftLeftBatch shifts the bank left by the next slice's width, then
// AssembleFromColumn ORs in (src >> (origW - end)) & mask
// (src/column.h:105-180, 208-1060; loop at src/stitch_composer.cpp:655-703).
// That reads and writes the bank once per slice.  Here every thread owns four
// consecutive rows, reads each source slice with one vector load per row
// group, folds the slices in registers and writes the bank once: the kernel
// moves exactly sum(source bytes) + bank bytes per row.
#include "device_common.cuh"
#include "fmcs_internal.h"

#include <algorithm>
#include <type_traits>

namespace fmcs {

namespace {

// One slice, ready to fold into a 64-bit bank value.  Sources of up to 4 bytes:
// ((value >> rshift) & mask) * mul, mul = 2^pos, added to the value (pos < 32) or
// mul = 2^(pos - 32), added to its high word: a shift, a mask and one
// multiply-add a row.  8-byte sources: the value shifted left by `shift` (right
// when negative) and masked to the bank bits the slice fills.
struct FoldSlice {
    const void *src;
    uint32_t src_bytes;
    uint32_t rshift, mask, mul;
    int high;
    int shift;
    uint32_t mlo, mhi;
};

struct StitchParams {
    FoldSlice s[kMaxSlices];
    int ns;
    uint32_t flip_lo, flip_hi;   // the bits of descending columns
};

constexpr int kStitchCtas = 4;   // resident CTAs per SM

// Rows of a group of four, and where a lane's groups start.  VEC: neighbours,
// moved by vectors.  Else (some array off a 16-byte boundary) 32 apart, so that a
// warp's lanes still read and write neighbours: the 32 groups of a warp hold its
// 128 rows either way.  (Four neighbours a lane, one access each: 16M rows of
// 1 + 2 + 4 bytes into 4 took 117 us, 79 so.)
template <bool VEC>
struct Group4 {
    static constexpr uint32_t kStep = VEC ? 1u : 32u;
    static __device__ __forceinline__ uint64_t first_row(uint64_t g) { return VEC ? g * 4 : (g & ~31ull) * 4 + (g & 31u); }
};

// Four rows of one slice as they come from memory: MAXB (the widest source's
// bytes per row) words.
template <int MAXB>
struct Raw4 {
    uint32_t w[MAXB];
};

// VEC: one vector load (the rows are whole and the source is aligned); else
// row by row (Group4), zero past n.
template <int MAXB, bool VEC>
__device__ __forceinline__ void load_raw(const void *base, uint32_t bytes, uint64_t row, uint64_t n, Raw4<MAXB> &r)
{
    if constexpr (!VEC) {
        // (the width is looked at once, so that the four loads are in flight together)
        auto four = [&](auto *p, auto &&put) {
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const uint64_t at = row + k * Group4<VEC>::kStep;
                put(k, at < n ? p[at] : 0u);
            }
        };
        if (bytes == 8) {
            if constexpr (MAXB >= 8)
                four((const uint64_t *)base, [&](int k, uint64_t v) {
                    r.w[2 * k] = (uint32_t)v;
                    r.w[2 * k + 1] = (uint32_t)(v >> 32);
                });
        } else if (bytes == 4) {
            if constexpr (MAXB >= 4) four((const uint32_t *)base, [&](int k, uint32_t v) { r.w[k] = v; });
        } else {
            r.w[0] = 0;
            if (bytes == 2) {
                r.w[1] = 0;
                four((const uint16_t *)base, [&](int k, uint32_t v) { r.w[k >> 1] |= v << (16 * (k & 1)); });
            } else {
                four((const uint8_t *)base, [&](int k, uint32_t v) { r.w[0] |= v << (8 * k); });
            }
        }
        return;
    }
    if constexpr (MAXB >= 8) {
        if (bytes == 8) {
            const uint4 *p = reinterpret_cast<const uint4 *>((const uint64_t *)base + row);
            const uint4 a = p[0], b = p[1];
            r.w[0] = a.x; r.w[1] = a.y; r.w[2] = a.z; r.w[3] = a.w;
            r.w[4] = b.x; r.w[5] = b.y; r.w[6] = b.z; r.w[7] = b.w;
            return;
        }
    }
    if constexpr (MAXB >= 4) {
        if (bytes == 4) {
            const uint4 a = *reinterpret_cast<const uint4 *>((const uint32_t *)base + row);
            r.w[0] = a.x; r.w[1] = a.y; r.w[2] = a.z; r.w[3] = a.w;
            return;
        }
    }
    if (bytes == 2) {
        const uint2 a = *reinterpret_cast<const uint2 *>((const uint16_t *)base + row);
        r.w[0] = a.x; r.w[1] = a.y;
    } else {
        r.w[0] = *reinterpret_cast<const uint32_t *>((const uint8_t *)base + row);
    }
}

// Folds a slice of four rows into their banks.
template <int MAXB>
__device__ __forceinline__ void fold(const FoldSlice &s, const Raw4<MAXB> &r, uint64_t (&acc)[4])
{
    if constexpr (MAXB >= 8) {
        if (s.src_bytes == 8) {
            const uint64_t m = (uint64_t)s.mhi << 32 | s.mlo;
            uint64_t v[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) v[k] = (uint64_t)r.w[2 * k] | ((uint64_t)r.w[2 * k + 1] << 32);
            if (s.shift > 0) {
#pragma unroll
                for (int k = 0; k < 4; ++k) v[k] <<= s.shift;
            } else if (s.shift < 0) {
#pragma unroll
                for (int k = 0; k < 4; ++k) v[k] >>= -s.shift;
            }
#pragma unroll
            for (int k = 0; k < 4; ++k) acc[k] |= v[k] & m;
            return;
        }
    }
    uint32_t x[4];
    if (MAXB >= 4 && s.src_bytes == 4) {
#pragma unroll
        for (int k = 0; k < 4; ++k) x[k] = (r.w[MAXB >= 4 ? k : 0] >> s.rshift) & s.mask;
    } else if (s.src_bytes == 2) {
        const uint32_t odd = s.rshift + 16;
#pragma unroll
        for (int k = 0; k < 4; ++k) x[k] = (r.w[k >> 1] >> (k & 1 ? odd : s.rshift)) & s.mask;
    } else {
#pragma unroll
        for (int k = 0; k < 4; ++k) x[k] = (r.w[0] >> (s.rshift + 8 * k)) & s.mask;
    }
    if (s.high) {
#pragma unroll
        for (int k = 0; k < 4; ++k) acc[k] += (uint64_t)(x[k] * s.mul) << 32;
    } else {
#pragma unroll
        for (int k = 0; k < 4; ++k) acc[k] += (uint64_t)x[k] * s.mul;
    }
}

template <typename B, bool VEC>
__device__ __forceinline__ void store4(B *bank, uint64_t row, uint64_t n, const uint64_t (&a)[4])
{
    if constexpr (VEC) {
        if constexpr (sizeof(B) == 1) {
            *reinterpret_cast<uint32_t *>(bank + row) = ((uint32_t)a[0] & 0xFF) | ((uint32_t)a[1] & 0xFF) << 8 |
                                                        ((uint32_t)a[2] & 0xFF) << 16 | (uint32_t)a[3] << 24;
        } else if constexpr (sizeof(B) == 2) {
            *reinterpret_cast<uint2 *>(bank + row) = make_uint2(((uint32_t)a[0] & 0xFFFF) | (uint32_t)a[1] << 16,
                                                                ((uint32_t)a[2] & 0xFFFF) | (uint32_t)a[3] << 16);
        } else if constexpr (sizeof(B) == 4) {
            *reinterpret_cast<uint4 *>(bank + row) =
                make_uint4((uint32_t)a[0], (uint32_t)a[1], (uint32_t)a[2], (uint32_t)a[3]);
        } else {
            ulonglong2 *p = reinterpret_cast<ulonglong2 *>(bank + row);
            p[0] = make_ulonglong2(a[0], a[1]);
            p[1] = make_ulonglong2(a[2], a[3]);
        }
    } else {
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const uint64_t at = row + k * Group4<VEC>::kStep;
            if (at < n) bank[at] = (B)a[k];
        }
    }
}

// With top_hist the kernel also counts the first radix level's digits: a CTA
// takes a contiguous run of units, part_groups groups of 4 rows of one chunk
// each (parts units a chunk), and adds a unit's counts to the chunk's 256-word
// row and to the chunk's super row after the chunks' rows.  Two shared
// histograms alternate by unit, so one is written out while the next unit
// loads.  Without, the groups are spread grid-stride.
//
// Each thread takes two groups of 4 rows per step, a stride apart; all slices
// of a batch (kBatch, by MAXB, the widest source's bytes, so that nothing
// spills) are loaded before the first is folded.
// Bound: HBM for few slices (16.8M rows of u32 + u64 into a u64 bank, 20 bytes a
// row: 66 us, 72 before), instructions for many (40M rows of five narrow
// columns into 8 bytes and one into 2: 227 us, 354 when every slice was
// shifted and masked in 64 bits a row).  More or fewer resident CTAs (3, 5) and
// 8-byte slices two at a time: within 10% either way, by case.
template <typename B, int MAXB, bool VEC>
__global__ void __launch_bounds__(256, kStitchCtas) stitch_kernel(const __grid_constant__ StitchParams p, B *bank,
                                                                  uint64_t n, uint32_t *top_hist,
                                                                  uint32_t hist_lo, uint32_t hist_mask,
                                                                  uint64_t chunk_groups, uint32_t part_groups,
                                                                  uint32_t parts, uint32_t units)
{
    kernel_prologue();
    constexpr int kBatch = MAXB == 8 ? 1 : MAXB == 4 ? 3 : 4;
    __shared__ uint32_t sh[2][256];
    const uint64_t groups = VEC ? n / 4 : (n + 127) / 128 * 32;
    auto count = [&](const uint64_t (&a)[4], uint64_t row, uint32_t *hist) {
        uint32_t d[4];
        if (hist_lo >= 32) {
#pragma unroll
            for (int k = 0; k < 4; ++k) d[k] = (uint32_t)(a[k] >> 32) >> (hist_lo - 32);
        } else {
#pragma unroll
            for (int k = 0; k < 4; ++k) d[k] = (uint32_t)(a[k] >> hist_lo);
        }
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if (VEC || row + k * Group4<VEC>::kStep < n) atomicAdd(&hist[d[k] & hist_mask], 1u);
    };
    auto step = [&](uint64_t g, uint64_t stride, uint64_t g_end, uint32_t *hist) {
        const bool two = g + stride < g_end;
        // (a lone group is folded twice)
        const uint64_t row0 = Group4<VEC>::first_row(g), row1 = Group4<VEC>::first_row(two ? g + stride : g);
        uint64_t a0[4] = {0, 0, 0, 0}, a1[4] = {0, 0, 0, 0};
#pragma unroll 1
        for (int s0 = 0; s0 < p.ns; s0 += kBatch) {
            Raw4<MAXB> r0[kBatch], r1[kBatch];
#pragma unroll
            for (int i = 0; i < kBatch; ++i) {
                if (s0 + i < p.ns) {
                    load_raw<MAXB, VEC>(p.s[s0 + i].src, p.s[s0 + i].src_bytes, row0, n, r0[i]);
                    load_raw<MAXB, VEC>(p.s[s0 + i].src, p.s[s0 + i].src_bytes, row1, n, r1[i]);
                }
            }
#pragma unroll
            for (int i = 0; i < kBatch; ++i) {
                if (s0 + i < p.ns) {
                    fold<MAXB>(p.s[s0 + i], r0[i], a0);
                    fold<MAXB>(p.s[s0 + i], r1[i], a1);
                }
            }
        }
        if (p.flip_lo | p.flip_hi) {
            const uint64_t flip = (uint64_t)p.flip_hi << 32 | p.flip_lo;
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                a0[k] ^= flip;
                a1[k] ^= flip;
            }
        }
        store4<B, VEC>(bank, row0, n, a0);
        if (hist) count(a0, row0, hist);
        if (two) {
            store4<B, VEC>(bank, row1, n, a1);
            if (hist) count(a1, row1, hist);
        }
    };
    // the rows past the last whole group of an aligned bank, a thread each
    auto tail = [&](uint32_t *hist) {
        const uint64_t row = (n & ~3ull) + threadIdx.x;
        if (!VEC || row >= n) return;
        uint64_t acc = 0;
        for (int s = 0; s < p.ns; ++s) {
            const FoldSlice &f = p.s[s];
            uint64_t v;
            switch (f.src_bytes) {
            case 1: v = ((const uint8_t *)f.src)[row]; break;
            case 2: v = ((const uint16_t *)f.src)[row]; break;
            case 4: v = ((const uint32_t *)f.src)[row]; break;
            default: v = ((const uint64_t *)f.src)[row]; break;
            }
            acc |= (f.shift >= 0 ? v << f.shift : v >> -f.shift) & ((uint64_t)f.mhi << 32 | f.mlo);
        }
        acc ^= (uint64_t)p.flip_hi << 32 | p.flip_lo;
        bank[row] = (B)acc;
        if (hist) atomicAdd(&hist[(uint32_t)(acc >> hist_lo) & hist_mask], 1u);
    };
    if (!top_hist) {
        const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
        for (uint64_t g = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; g < groups; g += 2 * stride)
            step(g, stride, groups, nullptr);
        if (blockIdx.x == 0) tail(nullptr);
        return;
    }
    sh[0][threadIdx.x] = 0;
    sh[1][threadIdx.x] = 0;
    const uint32_t per = (units + gridDim.x - 1) / gridDim.x;
    const uint32_t u0 = blockIdx.x * per, u1 = min(units, u0 + per);
    const uint32_t chunks = units / parts;
    __syncthreads();
    for (uint32_t u = u0; u <= u1; ++u) {
        const uint32_t set = (u - u0) & 1u;
        if (u < u1) {
            const uint32_t c = u / parts;
            const uint64_t g0 = c * chunk_groups + (uint64_t)(u % parts) * part_groups;
            const uint64_t g1 = min(min(groups, (c + 1) * chunk_groups), g0 + part_groups);
            for (uint64_t g = g0 + threadIdx.x; g < g1; g += 512) step(g, 256, g1, sh[set]);
            if (u + 1 == units) tail(sh[set]);
        }
        if (u > u0) {   // the unit before, counted in the other set
            const uint32_t v = sh[set ^ 1u][threadIdx.x];
            if (v) {
                const uint32_t c = (u - 1) / parts;
                atomicAdd(&top_hist[c * 256ull + threadIdx.x], v);
                atomicAdd(&top_hist[(chunks + c / kTopSuper) * 256ull + threadIdx.x], v);
                sh[set ^ 1u][threadIdx.x] = 0;
            }
        }
        __syncthreads();
    }
}

// Slice-at-a-time primitives (the reference's ShiftLeftBatch / AssembleFromColumn).
template <typename B>
__global__ void __launch_bounds__(256) bank_update_kernel(B *bank, uint64_t n, uint32_t lshift, const void *src,
                                                          uint32_t src_bytes, uint32_t rshift, uint32_t width)
{
    kernel_prologue();
    const uint64_t mask = width >= 64 ? ~0ull : ((1ull << width) - 1);
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        if (!src) {
            bank[i] = lshift >= 8 * sizeof(B) ? B(0) : (B)((uint64_t)bank[i] << lshift);
        } else {
            uint64_t v;
            switch (src_bytes) {
            case 1: v = ((const uint8_t *)src)[i]; break;
            case 2: v = ((const uint16_t *)src)[i]; break;
            case 4: v = ((const uint32_t *)src)[i]; break;
            default: v = ((const uint64_t *)src)[i]; break;
            }
            bank[i] = (B)((uint64_t)bank[i] | ((v >> rshift) & mask));
        }
    }
}

}  // namespace

int launch_bank_update(fmcs_ctx *ctx, void *bank, uint32_t bank_bytes, uint64_t n, uint32_t lshift,
                       const void *src, uint32_t src_bytes, uint32_t rshift, uint32_t width)
{
    if (n == 0) return FMCS_OK;
    const unsigned grid = (unsigned)std::min<uint64_t>((n + 255) / 256, (uint64_t)ctx->num_sms * 8);
    LaunchScope ls_(ctx, src ? "assemble" : "shift_left");
    switch (bank_bytes) {
    case 1: launch_k(bank_update_kernel<uint8_t>, grid, 256, 0, ctx->stream,
                     (uint8_t *)bank, n, lshift, src, src_bytes, rshift, width); break;
    case 2: launch_k(bank_update_kernel<uint16_t>, grid, 256, 0, ctx->stream,
                     (uint16_t *)bank, n, lshift, src, src_bytes, rshift, width); break;
    case 4: launch_k(bank_update_kernel<uint32_t>, grid, 256, 0, ctx->stream,
                     (uint32_t *)bank, n, lshift, src, src_bytes, rshift, width); break;
    case 8: launch_k(bank_update_kernel<uint64_t>, grid, 256, 0, ctx->stream,
                     (uint64_t *)bank, n, lshift, src, src_bytes, rshift, width); break;
    default: return set_error(ctx, FMCS_E_INVAL, "bank_bytes must be 1, 2, 4 or 8");
    }
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? FMCS_OK : cuda_fail(ctx, e, "bank update launch");
}

int launch_stitch(fmcs_ctx *ctx, const StitchSlice *sl, int ns, void *bank, uint32_t bank_bytes,
                  uint64_t n, uint32_t *top_hist, uint32_t key_bits, uint32_t chunk_rows, cudaStream_t stream)
{
    cudaStream_t st = stream ? stream : ctx->stream;
    if (ns < 1 || ns > kMaxSlices) return set_error(ctx, FMCS_E_INVAL, "stitch: 1..32 slices");
    if (!(bank_bytes == 1 || bank_bytes == 2 || bank_bytes == 4 || bank_bytes == 8))
        return set_error(ctx, FMCS_E_INVAL, "stitch: bank_bytes must be 1, 2, 4 or 8");
    if (n == 0) return FMCS_OK;
    StitchParams p{};
    bool aligned = ((uintptr_t)bank % 16) == 0;
    uint32_t pos = 0;   // bank bits to the right of the slice
    uint64_t flips = 0;
    for (int i = ns - 1; i >= 0; --i) {
        const uint64_t mask = sl[i].width >= 64 ? ~0ull : ((1ull << sl[i].width) - 1);
        const uint64_t at = pos < 64 ? mask << pos : 0ull;   // (bits shifted out of the bank are dropped)
        FoldSlice &f = p.s[i];
        f.src = sl[i].src;
        f.src_bytes = sl[i].src_bytes;
        f.shift = at ? (int)pos - (int)sl[i].rshift : 0;
        f.mlo = (uint32_t)at;
        f.mhi = (uint32_t)(at >> 32);
        f.rshift = sl[i].rshift;
        f.mask = at ? (uint32_t)(at >> pos) : 0u;
        f.high = pos >= 32;
        f.mul = at ? 1u << (pos & 31) : 0u;
        if (sl[i].invert) flips |= at;
        pos = pos < 64 ? pos + sl[i].width : pos;
        aligned = aligned && ((uintptr_t)sl[i].src % 16) == 0;
    }
    uint32_t maxb = 0;
    for (int i = 0; i < ns; ++i) maxb = std::max(maxb, sl[i].src_bytes);
    p.ns = ns;
    p.flip_lo = (uint32_t)flips;
    p.flip_hi = (uint32_t)(flips >> 32);
    const uint64_t groups = (n + 3) / 4;
    uint64_t blocks = (groups + 255) / 256;
    const uint64_t cap = (uint64_t)ctx->num_sms * 8;
    if (blocks > cap) blocks = cap;
    uint32_t hist_lo = 0, hist_mask = 0;
    uint64_t chunk_groups = 0;
    uint32_t part_groups = 0, parts = 1, units = 0;
    if (top_hist) {
        if (chunk_rows < 4 || chunk_rows % 4)
            return set_error(ctx, FMCS_E_INVAL, "stitch: chunk rows must be a multiple of 4");
        const uint32_t width = key_bits < 8u ? key_bits : 8u;
        hist_lo = key_bits - width;
        hist_mask = (1u << width) - 1u;
        chunk_groups = chunk_rows / 4;
        // enough CTAs to fill the GPU, each at least two steps of its threads
        const uint64_t chunks = (n + chunk_rows - 1) / chunk_rows;
        parts = (uint32_t)std::max<uint64_t>(1, std::min<uint64_t>(cap / chunks, chunk_groups / 512));
        part_groups = (uint32_t)((chunk_groups + parts - 1) / parts);
        units = (uint32_t)(chunks * parts);
        blocks = std::min<uint64_t>(units, (uint64_t)ctx->num_sms * kStitchCtas);
        cudaMemsetAsync(top_hist, 0, (chunks + (chunks + kTopSuper - 1) / kTopSuper) * 256 * sizeof(uint32_t), st);
    }
    const unsigned grid = (unsigned)blocks;
    LaunchScope ls_(ctx, "stitch");
    auto launch = [&](auto *b) {
        using B = std::remove_pointer_t<decltype(b)>;
        auto *k = !aligned    ? (maxb <= 4 ? stitch_kernel<B, 4, false> : stitch_kernel<B, 8, false>)
                  : maxb <= 2 ? stitch_kernel<B, 2, true>
                  : maxb <= 4 ? stitch_kernel<B, 4, true>
                              : stitch_kernel<B, 8, true>;
        launch_k(k, grid, 256, 0, st, p, b, n, top_hist, hist_lo, hist_mask, chunk_groups, part_groups, parts,
                 units);
    };
    switch (bank_bytes) {
    case 1: launch((uint8_t *)bank); break;
    case 2: launch((uint16_t *)bank); break;
    case 4: launch((uint32_t *)bank); break;
    default: launch((uint64_t *)bank); break;
    }
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? FMCS_OK : cuda_fail(ctx, e, "stitch launch");
}

}  // namespace fmcs
