// Visibility records and their binning by the first cell of the footprint.
#pragma once

#include "common.cuh"

namespace stpgpu {

// Per-visibility record written by the prepass.  flags: bit0 conj(kernel)
// for the original item (w < 0), bit1 conj(kernel) for the mirrored item
// (-w < 0).  The visibility is stored conjugated when the half-plane
// conversion flipped it.  16-byte aligned (32 B single, 48 B double
// precision): two or three 16-byte loads.
template <typename R>
struct alignas(16) Item {
    R vr, vi, w;
    int32_t gcx, gcy;
    int16_t cpx, cpy;
    uint16_t plane;
    uint8_t good, flags;
};
static_assert(sizeof(Item<float>) == 32 && sizeof(Item<double>) == 48, "item record sizes");

template <typename R>
__device__ __forceinline__ void item_centre(const Item<R>& it, int mir, int N, int& cx, int& cy)
{
    cx = mir ? N - it.gcx : it.gcx;
    cy = mir ? N - it.gcy : it.gcy;
}

// W-plane of sorted position k: the last plane whose first position <= k.
__device__ __forceinline__ int plane_of(const int64_t* first, int P, int64_t k)
{
    int lo = 0, hi = P - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) / 2;
        if (first[mid] <= k)
            lo = mid;
        else
            hi = mid - 1;
    }
    return lo;
}

// ---------------------------------------------------------------- binning

// A footprint (item, mirror) becomes one entry per place where its K x K
// cells land in the grid after wrapping: the first cell (row0, col0) may lie
// up to K - 1 before the grid, and cells outside [0, rows) x [0, N) are not
// gridded.  Almost every item has one entry; footprints across a grid edge
// and the mirrored copies near v = 0 have more.  Entries are binned by
// (row0, col0) into 8 x 8 bins, `pad` bins before the first block on either
// axis, so the entries that reach a block are those of the block's own bin
// and of the `pad` bins before it on each axis; bins are numbered down the
// rows first, which makes them pad + 1 contiguous ranges of records.  An
// entry is stored once, whatever number of blocks it reaches (the tile lists
// of a binning by overlap hold about 2.1 records per item at K = 7).
constexpr int kBlk = 8;        // block edge in cells
constexpr int kEntrySlots = 4; // entries per item whose places the count pass keeps

struct BlockBins {
    int N, rows;  // grid columns and rows
    int pad;      // ceil((largest K - 1) / 8)
    int brn, bcn; // bins along the rows and along the columns
    int wrap_neg; // exact gridder: rows below 0 wrap to the top
    int support;  // without W-projection
    const int* plane_support;
    const uint16_t* plane16; // W-projection without the |w| sort: plane of each item (input order), else null
    const uint32_t* order;   // W-projection with the sort: input index of each item (items in |w| order), else null
    const int64_t* first;    // then the first item of each plane
    int P;
    const uint8_t* ts_of; // A-projection: time step per visibility (nullable)
    int ntimesteps;
    int64_t n;
    uint32_t* count;  // entries per bin
    uint32_t* cursor; // fill cursors, used when some item has more than kEntrySlots entries
    uint32_t* ranks;  // [kEntrySlots][n] place of an item's entries in their bins
    uint32_t* rank_overflow;
    const uint32_t* off; // first entry of each bin, and of each column of bins the end (brn + 1 per column)
};

// One entry.  geom: row0 and col0 modulo 1024 (10 bits each), the support
// (7 bits), conjugated W-kernel (bit 27), mirrored copy (bit 28).
// koff: W-projection, the entry's kernel in the expanded tables; separable
// kernels, cpy | cpx << 16 (offset indices); exact kernels, the visibility.
template <typename R>
struct alignas(16) GridRec {
    R vr, vi;
    uint32_t koff, geom;
};
static_assert(sizeof(GridRec<float>) == 16 && sizeof(GridRec<double>) == 32, "record sizes");

__device__ __forceinline__ int item_plane(const BlockBins& b, int64_t k)
{
    if (b.plane16)
        return b.plane16[k];
    if (!b.order)
        return 0;
    int plane = plane_of(b.first, b.P, k);
    if (b.ts_of)
        plane = plane * b.ntimesteps + b.ts_of[b.order[k]];
    return plane;
}

// f(row0, col0, bin column, bin row) for every entry of one footprint.
template <typename F>
__device__ __forceinline__ void for_entries(const BlockBins& b, int cx, int cy, int S, F f)
{
    const int K = 2 * S + 1;
    const int rb = cy - S, cb = cx - S;
#pragma unroll 1
    for (int ri = 0; ri < 3; ri++) {
        // in place; rows at or beyond N wrap once; rows below 0 wrap for the exact gridder
        if (ri == 1 && rb + K <= b.N)
            continue;
        if (ri == 2 && !(b.wrap_neg && rb < 0))
            continue;
        const int row0 = ri == 0 ? rb : (ri == 1 ? rb - b.N : rb + b.N);
        if (row0 >= b.rows || row0 + K <= 0)
            continue;
#pragma unroll 1
        for (int ci = 0; ci < 3; ci++) {
            if (ci == 1 && cb + K <= b.N)
                continue;
            if (ci == 2 && cb >= 0)
                continue;
            const int col0 = ci == 0 ? cb : (ci == 1 ? cb - b.N : cb + b.N);
            if (col0 >= b.N || col0 + K <= 0)
                continue;
            f(row0, col0, uint32_t(col0 + kBlk * b.pad) / kBlk, uint32_t(row0 + kBlk * b.pad) / kBlk);
        }
    }
}

// Counts one item's entries; the atomics return their places in the bins,
// kept for the fill pass.
template <typename R>
__device__ __forceinline__ void count_entries(const BlockBins& b, const Item<R>& it, int64_t k, int S)
{
    int q = 0;
    for (int mir = 0; mir < int(it.good); mir++) {
        int cx, cy;
        item_centre(it, mir, b.N, cx, cy);
        for_entries(b, cx, cy, S, [&](int, int, uint32_t bc, uint32_t br) {
            const uint32_t r = atomicAdd(&b.count[bc * uint32_t(b.brn) + br], 1u);
            if (q < kEntrySlots)
                b.ranks[size_t(q) * size_t(b.n) + size_t(k)] = r; // slot-major: coalesced
            else
                *b.rank_overflow = 1u;
            q++;
        });
    }
}

// W-projection: once the planes' supports are known (the prepass counts the
// entries of the other kernels).
template <typename R>
__global__ void __launch_bounds__(256) k_bin_count(BlockBins b, const Item<R>* __restrict__ items)
{
    const int64_t k = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (k >= b.n)
        return;
    const Item<R> it = items[k];
    if (it.good)
        count_entries(b, it, k, b.plane_support[item_plane(b, k)]);
}

// Exclusive sum over the block's threads; *total = the sum of all.
__device__ __forceinline__ uint32_t block_excl_sum(uint32_t v, uint32_t* total)
{
    __shared__ uint32_t wsum[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = int(blockDim.x >> 5);
    uint32_t x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o)
            x += y;
    }
    if (lane == 31)
        wsum[warp] = x;
    __syncthreads();
    uint32_t before = 0, all = 0;
    for (int w = 0; w < nw; w++) {
        if (w < warp)
            before += wsum[w];
        all += wsum[w];
    }
    __syncthreads();
    *total = all;
    return before + x - v;
}

// Offsets of the bins, one block per column of bins: the ranges that a block
// of cells reads never leave a column, so the columns' records may lie in any
// order and each takes its room from one cursor (*total, zeroed before; the
// entries in all afterwards).  One short launch where a scan over all bins
// takes two with a dependence along the bins.
__global__ void __launch_bounds__(256) k_bin_scan(const uint32_t* __restrict__ count, uint32_t* off, uint32_t* cursor,
    int brn, const uint32_t* rank_overflow, uint32_t* total)
{
    __shared__ uint32_t s_base;
    const uint32_t* c = count + size_t(blockIdx.x) * size_t(brn);
    uint32_t* o = off + size_t(blockIdx.x) * size_t(brn + 1);
    uint32_t sum = 0;
    for (int i = threadIdx.x; i < brn; i += blockDim.x)
        sum += c[i];
    uint32_t all;
    block_excl_sum(sum, &all);
    if (threadIdx.x == 0)
        s_base = atomicAdd(total, all);
    __syncthreads();
    uint32_t base = s_base;
    const bool clear = *rank_overflow != 0u; // the fill pass takes its places from the cursors
    for (int i0 = 0; i0 < brn; i0 += blockDim.x) {
        const int i = i0 + threadIdx.x;
        const uint32_t v = i < brn ? c[i] : 0u;
        uint32_t part;
        const uint32_t e = block_excl_sum(v, &part);
        if (i < brn) {
            o[i] = base + e;
            if (clear)
                cursor[size_t(blockIdx.x) * size_t(brn) + i] = 0u;
        }
        base += part;
    }
    if (threadIdx.x == 0)
        o[brn] = base;
}

// Records at their places.  The capacity holds every entry there can be
// (bit 1 of *err otherwise, never expected).
template <typename R>
struct BinFill {
    GridRec<R>* rec;
    R* wts; // weight per record (beam), nullable
    uint64_t cap;
    const uint32_t* wk_off; // W-projection: table offset per plane (x time step)
    int cs, os, exact;
    unsigned int* err;
};

template <typename R>
__global__ void __launch_bounds__(256) k_bin_fill(BlockBins b, const Item<R>* __restrict__ items, BinFill<R> q)
{
    const int64_t k = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (k >= b.n)
        return;
    const Item<R> it = items[k];
    if (!it.good)
        return;
    int S = b.support, plane = 0;
    if (b.plane_support) {
        plane = item_plane(b, k);
        S = b.plane_support[plane];
    }
    const int K = 2 * S + 1;
    const bool ranked = *b.rank_overflow == 0u;
    int e = 0;
    for (int mir = 0; mir < int(it.good); mir++) {
        int cx, cy;
        item_centre(it, mir, b.N, cx, cy);
        int cpx = it.cpx, cpy = it.cpy;
        if (mir && q.os > 1) {
            cpx = q.os - cpx;
            cpy = q.os - cpy;
        }
        GridRec<R> r;
        r.vr = it.vr * it.w;
        r.vi = (mir ? -it.vi : it.vi) * it.w;
        const uint32_t conj = (it.flags >> (mir ? 1 : 0)) & 1u;
        if (b.plane_support)
            r.koff = q.wk_off[plane] + uint32_t((cpy * q.cs + cpx) * K * K);
        else
            r.koff = q.exact ? uint32_t(k) : uint32_t(cpy) | (uint32_t(cpx) << 16);
        for_entries(b, cx, cy, S, [&](int row0, int col0, uint32_t bc, uint32_t br) {
            const uint32_t place = ranked ? b.ranks[size_t(e) * size_t(b.n) + size_t(k)]
                                          : atomicAdd(&b.cursor[bc * uint32_t(b.brn) + br], 1u);
            e++;
            r.geom = uint32_t(row0 & 1023) | (uint32_t(col0 & 1023) << 10) | (uint32_t(S) << 20) | (conj << 27)
                | (uint32_t(mir) << 28);
            const uint64_t pos = uint64_t(b.off[bc * uint32_t(b.brn + 1) + br]) + place;
            if (pos < q.cap) {
                q.rec[pos] = r;
                if (q.wts)
                    q.wts[pos] = it.w;
            } else {
                atomicOr(q.err, 1u);
            }
        });
    }
}

} // namespace stpgpu
