// Block gridder: binning of the footprints by their first cell and the
// output-stationary gridding kernels over 8 x 8 blocks of grid cells
// (gridder.h:596-994 for the gridding semantics).
#pragma once

#include "imager_kernels.cuh"

namespace stpgpu {

// ---------------------------------------------------------------- kernel tables

// The 1-D kernel table in rows of `tw` values with zeros around the K taps
// (tap d of offset c at [c * tw + d + 7]), so a block kernel indexes it
// without a range check, and a last row of zeros.
__global__ void k_pad_table(const double* k1d, int cs, int K, int tw, double* out)
{
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (cs + 1) * tw)
        return;
    const int c = t / tw, d = t % tw - 7;
    out[t] = c < cs && d >= 0 && d < K ? k1d[c * K + d] : 0.0;
}

// Exact gridder: the two 1-D kernels of every visibility, tab[k][axis][K]
// (axis 0: v, 1: u).  make_kernel_array divides the outer product by its
// sum (conv_func.h:279-303), which is the product of the two sums; the
// functors are even, so the mirrored copy reads them backwards.
__global__ void __launch_bounds__(256) k_exact_tables(int kf, double trunc, int S, const double* __restrict__ frac,
    int64_t n, double* __restrict__ tab)
{
    const int64_t t = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (t >= 2 * n)
        return;
    const int64_t k = t >> 1;
    const int axis = int(t & 1), K = 2 * S + 1;
    const double f = frac[(axis ? 0 : n) + k];
    double* o = tab + size_t(t) * K;
    double sum = 0.0;
    for (int i = 0; i < K; i++) {
        const double v = kernel_value(kf, trunc, (double(i) - S) - f);
        o[i] = v;
        sum += v;
    }
    for (int i = 0; i < K; i++)
        o[i] = o[i] / sum;
}

// ---------------------------------------------------------------- block gridder

// One warp per 8 x 8 block of cells, eight warps (64 rows x 8 columns) per
// CTA.  The cells stay in registers: nothing is read back, zeroed or
// updated in memory, and every cell of the grid is written exactly once.
//
// The CTA's entries are fetched and decoded once into shared memory
// (C::kCta at a time, footprints of up to 8 (kCtaBins - 1) + 1 cells): the bins of
// neighbouring blocks overlap, and a block that stages its own entries spends
// as much on its ranges and on decoding as on gridding when it holds a few
// tens of them (138 M warp instructions on the 1M-visibility headline call,
// 47 per entry and block, 26 of them the gridding).  Each warp then looks at
// the entries of its own bins 32 at a time, lists those that reach its block
// and hands the list to the core C.
//
// CTAs with a block of more than 2 kHeavy entries (the centre of a
// concentrated uv coverage) or, for W-kernels, with more than C::kCta in all,
// and those of wider footprints, take their entries block by block, 32 at a
// time through shared memory; blocks with more than kHeavy entries are then
// taken by all eight warps together, their partial cells summed in a fixed
// order.
constexpr int kGridWarps = 8;
constexpr uint32_t kHeavy = 512;
constexpr uint32_t kFew = 256; // entries of a column of blocks that its warps take on their own (sparse grids)
constexpr int kCtaBins = 5; // bins per axis that reach a block, at most, for staging by CTA

struct BlockRanges {
    uint32_t pre, delta; // lane j: entries before range j, and range j's first record minus that
    uint32_t total;
    int nb;
};

// Ranges of `len` entries from `beg` on, lane j's for j < nb <= 32, as one
// stream.
__device__ __forceinline__ BlockRanges make_ranges(uint32_t beg, uint32_t len, int nb)
{
    const int lane = threadIdx.x & 31;
    uint32_t incl = len;
    for (int o = 1; o < nb; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o)
            incl += y;
    }
    BlockRanges r;
    r.pre = incl - len;
    r.delta = beg - r.pre;
    r.total = __shfl_sync(0xffffffffu, incl, nb - 1);
    r.nb = nb;
    return r;
}

// Ranges j0 .. j0 + nb - 1 (nb <= 32) of block (br, bc): the bins' columns.
__device__ __forceinline__ BlockRanges block_ranges(const uint32_t* __restrict__ off, int brn, int br, int bc, int rows_nb,
    int nb)
{
    const int lane = threadIdx.x & 31;
    uint32_t beg = 0, len = 0;
    if (lane < nb) {
        const uint32_t* o = off + size_t(bc + lane) * size_t(brn + 1) + size_t(br);
        beg = o[0];
        len = o[rows_nb] - beg;
    }
    return make_ranges(beg, len, nb);
}

// Record of stream position t.
__device__ __forceinline__ uint32_t stream_record(const BlockRanges& r, uint32_t t)
{
    uint32_t d = __shfl_sync(0xffffffffu, r.delta, 0);
    for (int j = 1; j < r.nb; j++) {
        const uint32_t pj = __shfl_sync(0xffffffffu, r.pre, j), dj = __shfl_sync(0xffffffffu, r.delta, j);
        if (t >= pj)
            d = dj;
    }
    return t + d;
}

// Positions of the entries that reach a warp's block, in PARTS lists: an entry
// is on the list of every part of the block that it reaches, and the parts
// take an entry each at a time.  The longest list counts, which over 32
// entries (one bin's, often) is that of the part next to it, so two lists
// gather entries over several rounds before they are added; one list is added
// after each round.  Lists are filled up with a dummy to a multiple of four.
template <int PARTS>
struct BlockList {
    static constexpr int kSize = PARTS > 1 ? 128 : 32;
    uint16_t* list;
    int m[PARTS];
};

// The entries listed added to the block whose first cell is (row, col)
// (relative to the staged entries' origin).
template <class C, int PARTS>
__device__ __forceinline__ void list_add(const typename C::Params& p, const double* stab, const typename C::Staged* st,
    uint32_t dummy, int row, int col, BlockList<PARTS>& b, typename C::A (&acc)[C::NACC])
{
    const int lane = threadIdx.x & 31;
    int n = b.m[0];
#pragma unroll
    for (int h = 1; h < PARTS; h++)
        n = max(n, b.m[h]);
    n = (n + 3) & ~3;
#pragma unroll
    for (int h = 0; h < PARTS; h++)
        for (int i = b.m[h] + lane; i < n; i += 32)
            b.list[h * BlockList<PARTS>::kSize + i] = uint16_t(dummy);
    __syncwarp();
    C::template accumulate<PARTS>(p, stab, st, b.list, n, row, col, acc);
    __syncwarp();
#pragma unroll
    for (int h = 0; h < PARTS; h++)
        b.m[h] = 0;
}

// Entries of st, one per lane (position `at`, if `valid`), listed if they
// reach the block, and added if they are the only list's or a list may not
// have room for 32 more.
template <class C, int PARTS>
__device__ __forceinline__ void block_add(const typename C::Params& p, const double* stab, const typename C::Staged* st,
    uint32_t at, bool valid, uint32_t dummy, int row, int col, BlockList<PARTS>& b, typename C::A (&acc)[C::NACC])
{
    const int lane = threadIdx.x & 31;
    unsigned reach = 0; // bit h: part h
    bool odd = false;
    if (valid) {
        const typename C::Staged& s = st[at];
        reach = C::template reach<PARTS>(p, s, row, col);
        odd = reach && C::odd(s);
    }
    bool full = PARTS == 1;
#pragma unroll
    for (int h = 0; h < PARTS; h++) {
        const bool in = ((reach >> h) & 1u) && !odd;
        const unsigned mask = __ballot_sync(0xffffffffu, in);
        if (in)
            b.list[h * BlockList<PARTS>::kSize + b.m[h] + __popc(mask & ((1u << lane) - 1u))] = uint16_t(at);
        b.m[h] += __popc(mask);
        full |= b.m[h] > BlockList<PARTS>::kSize - 32;
    }
    if (C::kOdd) {
        unsigned o = __ballot_sync(0xffffffffu, odd);
        for (; o; o &= o - 1)
            C::add_odd(p, stab, st[__shfl_sync(0xffffffffu, at, __ffs(int(o)) - 1)], row, col, acc);
    }
    if (full)
        list_add<C, PARTS>(p, stab, st, dummy, row, col, b, acc);
}

template <class C>
__device__ __forceinline__ void block_walk(const typename C::Params& p, const double* stab, const BlockRanges& r, int r0,
    int c0, int first, int stride, typename C::Staged* st, BlockList<1>& list, typename C::A (&acc)[C::NACC])
{
    const int lane = threadIdx.x & 31;
    uint32_t t = uint32_t(first) * 32u;
    typename C::Raw raw {};
    if (t < r.total) {
        const uint32_t i = stream_record(r, t + lane);
        if (t + lane < r.total)
            raw = C::fetch(p, i);
    }
    while (t < r.total) {
        const uint32_t n = min(32u, r.total - t);
        if (uint32_t(lane) < n)
            st[lane] = C::decode(p, raw, r0, c0);
        __syncwarp();
        // the next 32 records are in flight while these are gridded
        const uint32_t tn = t + uint32_t(stride) * 32u;
        if (tn < r.total) {
            const uint32_t i = stream_record(r, tn + lane);
            if (tn + lane < r.total)
                raw = C::fetch(p, i);
        }
        block_add<C, 1>(p, stab, st, uint32_t(lane), uint32_t(lane) < n, 32, 0, 0, list, acc);
        t = tn;
    }
}

using CtaOffsets = uint32_t[kGridWarps + kCtaBins]; // of one column of bins

// The `total` entries of the blocks in column bc (bins at off, nb to an axis), staged at `all`.
template <class C, int PARTS>
__device__ __forceinline__ void grid_staged(const typename C::Params& p, const double* stab, typename C::Staged* all,
    const CtaOffsets* off, uint16_t* lists, int bc, int nb, uint32_t total)
{
    using A = typename C::A;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int br0 = int(blockIdx.x) * kGridWarps, br = br0 + warp;
    const int no = kGridWarps + nb;
    const uint32_t dummy = C::kCta + uint32_t(warp);
    BlockList<PARTS> list { lists, {} };
    if (threadIdx.x < kGridWarps)
        all[C::kCta + threadIdx.x] = C::dummy(p, int(threadIdx.x) * kBlk, 0);
    // lane j < nb: column j's entries in the CTA's order, all and the warp's
    uint32_t beg = 0, end = 0;
    {
        const uint32_t o = lane < nb ? off[lane][0] : 0u;
        const BlockRanges c = make_ranges(0, lane < nb ? off[lane][no - 1] - o : 0u, nb);
        if (lane < nb) {
            beg = c.pre + off[lane][warp] - o;
            end = c.pre + off[lane][warp + nb] - o;
        }
    }
    A acc[C::NACC] = {};
    uint32_t w0 = 0;
    for (;;) {
        const uint32_t w1 = C::kWindows ? min(total, w0 + C::kCta) : total;
        for (uint32_t t = w0 + threadIdx.x; t < w1; t += 32 * kGridWarps) {
            uint32_t i = t, j = 0;
            for (;; j++) {
                const uint32_t len = off[j][no - 1] - off[j][0];
                if (i < len)
                    break;
                i -= len;
            }
            all[t - w0] = C::decode(p, C::fetch(p, off[j][0] + i), br0 * kBlk, bc * kBlk);
        }
        __syncthreads();
        const uint32_t lo = C::kWindows ? max(beg, w0) : beg, hi = C::kWindows ? min(end, w1) : end;
        const BlockRanges r = make_ranges(lo - w0, hi > lo ? hi - lo : 0u, nb);
        for (uint32_t t = 0; t < r.total; t += 32)
            block_add<C, PARTS>(p, stab, all, stream_record(r, t + lane), t + lane < r.total, dummy, warp * kBlk, 0, list,
                acc);
        if (PARTS > 1)
            list_add<C, PARTS>(p, stab, all, dummy, warp * kBlk, 0, list, acc);
        if (!C::kWindows || w1 == total)
            break;
        w0 = w1;
        __syncthreads(); // the window's entries are gridded
    }
    if (br < (p.rows + kBlk - 1) / kBlk)
        C::template store<PARTS>(p, br * kBlk, bc * kBlk, acc);
}

// Zeros in 8 columns of 64 cells, a column per warp.
template <class C>
__device__ __forceinline__ void store_zeros(const typename C::Params& p, int r0, int c0)
{
    const int c = c0 + int(threadIdx.x >> 5);
    if (c >= p.N)
        return;
#pragma unroll
    for (int k = 0; k < kGridWarps * kBlk / 32; k++) {
        const int r = r0 + 32 * k + int(threadIdx.x & 31);
        if (r < p.rows)
            C::store_zero(p, size_t(c) * size_t(p.ld) + size_t(r));
    }
}

// The blocks of column bc taken one by one, each warp's entries 32 at a time.
template <class C>
__device__ __forceinline__ void grid_unstaged(const typename C::Params& p, const double* stab, unsigned char* smem,
    uint16_t (*s_list)[C::kParts * BlockList<C::kParts>::kSize], uint32_t& s_heavy, int bc, int nb, int skip)
{
    using A = typename C::A;
    using Staged = typename C::Staged;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int nbr = (p.rows + kBlk - 1) / kBlk;
    const int br0 = int(blockIdx.x) * kGridWarps, br = br0 + warp;
    Staged* st = reinterpret_cast<Staged*>(smem) + warp * 33;
    BlockList<1> list { s_list[warp], {} };
    if (lane == 0)
        st[32] = C::dummy(p, 0, 0);
    if (threadIdx.x == 0)
        s_heavy = 0;
    __syncthreads();
    if (br < nbr) {
        A acc[C::NACC] = {};
        uint32_t total = 0;
        bool heavy = false;
        // at most 32 ranges at a time (33 for the largest supports)
        for (int j = 0; j < nb; j += 32) {
            const BlockRanges r = block_ranges(p.off, p.brn, br + skip, bc + skip + j, nb, min(nb - j, 32));
            total += r.total;
            heavy = total > kHeavy;
            if (heavy)
                break;
            block_walk<C>(p, stab, r, br * kBlk, bc * kBlk, 0, 1, st, list, acc);
        }
        if (heavy) {
            if (lane == 0)
                atomicOr(&s_heavy, 1u << warp);
        } else {
            C::template store<1>(p, br * kBlk, bc * kBlk, acc);
        }
    }
    __syncthreads();
    for (uint32_t h = s_heavy; h; h &= h - 1) {
        const int hw = __ffs(int(h)) - 1;
        const int hbr = br0 + hw;
        A acc[C::NACC] = {};
        for (int j = 0; j < nb; j += 32) {
            const BlockRanges r = block_ranges(p.off, p.brn, hbr + skip, bc + skip + j, nb, min(nb - j, 32));
            block_walk<C>(p, stab, r, hbr * kBlk, bc * kBlk, warp, kGridWarps, st, list, acc);
        }
        __syncthreads(); // the staged records are read; the same memory takes the partial cells
        A* red = reinterpret_cast<A*>(smem);
        for (int q = 0; q < C::NACC; q++)
            red[(q * kGridWarps + warp) * 32 + lane] = acc[q];
        __syncthreads();
        if (warp == hw) {
            for (int q = 0; q < C::NACC; q++) {
                A v = A(0);
                for (int w = 0; w < kGridWarps; w++)
                    v += red[(q * kGridWarps + w) * 32 + lane];
                acc[q] = v;
            }
            C::template store<1>(p, hbr * kBlk, bc * kBlk, acc);
        }
        __syncthreads();
        if (lane == 0)
            st[32] = C::dummy(p, 0, 0); // overwritten by the partial cells
        __syncwarp();
    }
}

// The blocks of column bc on their own: each warp's few entries without a
// barrier (the ranges from the CTA's offsets).
template <class C>
__device__ __forceinline__ void grid_few(const typename C::Params& p, const double* stab, typename C::Staged* st,
    uint16_t* s_list, const CtaOffsets* off, int br, int bc, int nb)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (br >= (p.rows + kBlk - 1) / kBlk)
        return;
    uint32_t beg = 0, len = 0;
    if (lane < nb) {
        beg = off[lane][warp];
        len = off[lane][warp + nb] - beg;
    }
    typename C::A acc[C::NACC] = {};
    if (__any_sync(0xffffffffu, len != 0)) {
        if (lane == 0)
            st[32] = C::dummy(p, 0, 0);
        BlockList<1> list { s_list, {} };
        block_walk<C>(p, stab, make_ranges(beg, len, nb), br * kBlk, bc * kBlk, 0, 1, st, list, acc);
    }
    C::template store<1>(p, br * kBlk, bc * kBlk, acc);
}

// kFewCols blocks beside each other: where the warp has at most 32 entries for
// all of them, these are fetched and decoded once.
constexpr int kFewCols = 4;
template <class C>
__device__ __forceinline__ void grid_few_columns(const typename C::Params& p, const double* stab, typename C::Staged* st,
    uint16_t* s_list, const CtaOffsets* off, int br, int bc, int nb)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (br >= (p.rows + kBlk - 1) / kBlk)
        return;
    uint32_t beg = 0, len = 0;
    if (lane < nb + kFewCols - 1) {
        beg = off[lane][warp];
        len = off[lane][warp + nb] - beg;
    }
    const BlockRanges r = make_ranges(beg, len, nb + kFewCols - 1);
    if (r.total > 32) {
#pragma unroll 1
        for (int k = 0; k < kFewCols; k++)
            grid_few<C>(p, stab, st, s_list, off + k, br, bc + k, nb);
        return;
    }
    const bool valid = uint32_t(lane) < r.total;
    if (r.total > 0) {
        const uint32_t i = stream_record(r, lane);
        if (valid)
            st[lane] = C::decode(p, C::fetch(p, i), br * kBlk, bc * kBlk);
    }
    BlockList<1> list { s_list, {} };
#pragma unroll 1
    for (int k = 0; k < kFewCols; k++) {
        typename C::A acc[C::NACC] = {};
        if (r.total > 0) {
            if (lane == 0)
                st[32] = C::dummy(p, 0, k * kBlk);
            __syncwarp();
            block_add<C, 1>(p, stab, st, uint32_t(lane), valid, 32, 0, k * kBlk, list, acc);
        }
        C::template store<1>(p, br * kBlk, (bc + k) * kBlk, acc);
    }
    __syncwarp();
}

// COLS: columns of blocks that a CTA takes one after the other.  One, except
// on sparse grids, where most blocks only get their zeros or a few entries: a
// CTA for each column of eight blocks is then bound by its launch, the latency
// of its offsets and its barriers.  Eight columns share the offsets, empty
// ones are stored at once, and up to kFew entries are taken without a barrier
// (64 instead of 256: 48 against 44 us for 65k normally distributed
// visibilities on 4096^2).  What is left is bound by the instructions that a
// block costs whatever it holds (74 % of the issue slots), hence four columns
// at once (135 -> 99 us below); fetching the next column's records ahead gave
// nothing.  Kernel with one column and eight, disk coverage, single-precision
// cells: 26k visibilities on 8192^2 169 and 83 us, 157k 203 and 99, with
// W-kernels 260 and 127; 56k on 12000^2 357 and 166.
template <class C, int COLS>
__global__ void __launch_bounds__(32 * kGridWarps, C::kMinBlocks) k_grid_blocks(const __grid_constant__ typename C::Params p)
{
    using A = typename C::A;
    using Staged = typename C::Staged;
    // entries of the CTA and a dummy per warp; or 32 and a dummy per warp; or
    // the partial cells of a block taken by all warps
    constexpr size_t kStage = sizeof(Staged) * (C::kCta + kGridWarps);
    constexpr size_t kRed = sizeof(A) * C::NACC * 32 * kGridWarps;
    static_assert(C::kCta + kGridWarps >= 33 * kGridWarps, "staging by warp");
    __shared__ __align__(16) unsigned char smem[kStage > kRed ? kStage : kRed];
    __shared__ uint16_t s_list[kGridWarps][C::kParts * BlockList<C::kParts>::kSize];
    __shared__ CtaOffsets s_off[kCtaBins + COLS - 1];
    __shared__ uint32_t s_heavy;
    const int warp = threadIdx.x >> 5;
    Staged* all = reinterpret_cast<Staged*>(smem);
    const int br0 = int(blockIdx.x) * kGridWarps, bc0 = int(blockIdx.y) * COLS;
    const int nb = C::bins(p);       // bins that reach a block on either axis
    const int skip = p.pad + 1 - nb; // (those further away cannot)
    const int cols = COLS == 1 ? 1 : min(COLS, (p.N + kBlk - 1) / kBlk - bc0);
    __shared__ double s_tab[C::kTab > 0 ? C::kTab : 1];
    const double* stab = s_tab;
    const int no = kGridWarps + nb;
    if (nb <= kCtaBins) {
        // s_off[j]: the offsets of the CTA's bins in column j
        for (int t = threadIdx.x; t < (nb + cols - 1) * no; t += 32 * kGridWarps) {
            const int j = t / no, i = t - j * no;
            s_off[j][i] = p.off[size_t(bc0 + skip + j) * size_t(p.brn + 1) + size_t(min(br0 + skip + i, p.brn))];
        }
        if (COLS > 1)
            C::load_table(p, s_tab);
        __syncthreads();
    } else if (COLS > 1) {
        C::load_table(p, s_tab);
    }
    bool shared = false; // the column before was one of the whole CTA
    uint32_t totals = 1; // lane k: entries of column k
    if (nb <= kCtaBins) {
        const int lane = threadIdx.x & 31, k = COLS == 1 ? 0 : min(lane, cols - 1);
        totals = 0;
        for (int j = 0; j < nb; j++)
            totals += s_off[k + j][no - 1] - s_off[k + j][0];
    }
    const unsigned few = COLS == 1 || nb > kCtaBins ? 0u : __ballot_sync(0xffffffffu, totals <= kFew);
    const unsigned some = COLS == 1 ? 1u : __ballot_sync(0xffffffffu, totals != 0);
    for (int k = 0; k < cols; k++) {
        const int bc = bc0 + k;
        const CtaOffsets* off = s_off + k;
        if (COLS > 1 && k % kFewCols == 0 && k + kFewCols <= cols && ((~few >> k) & ((1u << kFewCols) - 1u)) == 0) {
            if (((some >> k) & ((1u << kFewCols) - 1u)) == 0) {
                for (int c = 0; c < kFewCols; c++)
                    store_zeros<C>(p, br0 * kBlk, (bc + c) * kBlk);
            } else {
                if (shared)
                    __syncthreads(); // the entries of the column before are gridded
                shared = false;
                grid_few_columns<C>(p, stab, all + warp * 33, s_list[warp], off, br0 + warp, bc, nb);
            }
            k += kFewCols - 1;
            continue;
        }
        const uint32_t total = COLS == 1 ? totals : __shfl_sync(0xffffffffu, totals, k);
        if (total == 0) { // nothing reaches the blocks: most of a grid outside the uv coverage
            store_zeros<C>(p, br0 * kBlk, bc * kBlk);
            continue;
        }
        if (COLS > 1) {
            if (shared)
                __syncthreads(); // the entries of the column before are gridded
            shared = total > kFew || nb > kCtaBins;
            if (!shared) {
                grid_few<C>(p, stab, all + warp * 33, s_list[warp], off, br0 + warp, bc, nb);
                continue;
            }
            __syncthreads(); // no warp is still at a column of its own
        } else {
            C::load_table(p, s_tab);
        }
        bool staged = false;
        if (nb <= kCtaBins) {
            uint32_t own = 0;
            if (C::kWindows)
                for (int j = 0; j < nb; j++)
                    own += off[j][warp + nb] - off[j][warp];
            // (with one column, the barrier also orders the table before its first use)
            staged = C::kWindows ? !__syncthreads_or(own > 2 * kHeavy) : total <= C::kCta;
        }
        if (!staged)
            grid_unstaged<C>(p, s_tab, smem, s_list, s_heavy, bc, nb, skip);
        else if (C::kParts > 1 && C::parts(p))
            grid_staged<C, C::kParts>(p, stab, all, off, s_list[warp], bc, nb, total);
        else
            grid_staged<C, 1>(p, stab, all, off, s_list[warp], bc, nb, total);
    }
}

// Dense grids: SPLIT warps share a block (every SPLIT-th 32 entries of its
// stream each) and sum their cells in a fixed order; a CTA has 8 / SPLIT
// blocks.  A small image with many visibilities has too few blocks to fill
// the GPU with one warp each, and along uv tracks most of its entries fall
// into a tenth of them.
template <class C, int SPLIT>
__global__ void __launch_bounds__(32 * kGridWarps) k_grid_dense(const __grid_constant__ typename C::Params p)
{
    using A = typename C::A;
    using Staged = typename C::Staged;
    constexpr size_t kStage = sizeof(Staged) * 33 * kGridWarps;
    constexpr size_t kRed = sizeof(A) * C::NACC * 32 * kGridWarps;
    __shared__ __align__(16) unsigned char smem[kStage > kRed ? kStage : kRed];
    __shared__ uint16_t s_list[kGridWarps][C::kParts * BlockList<C::kParts>::kSize];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int sub = warp % SPLIT, first = warp - sub;
    __shared__ double s_tab[C::kTab > 0 ? C::kTab : 1];
    const double* stab = s_tab;
    Staged* st = reinterpret_cast<Staged*>(smem) + warp * 33;
    BlockList<1> list { s_list[warp], {} };
    if (lane == 0)
        st[32] = C::dummy(p, 0, 0);
    C::load_table(p, s_tab);
    __syncthreads();
    const int nbr = (p.rows + kBlk - 1) / kBlk;
    const int br = int(blockIdx.x) * (kGridWarps / SPLIT) + warp / SPLIT, bc = int(blockIdx.y);
    const int nb = C::bins(p), skip = p.pad + 1 - nb;
    A acc[C::NACC] = {};
    if (br < nbr)
        for (int j = 0; j < nb; j += 32) {
            const BlockRanges r = block_ranges(p.off, p.brn, br + skip, bc + skip + j, nb, min(nb - j, 32));
            block_walk<C>(p, stab, r, br * kBlk, bc * kBlk, sub, SPLIT, st, list, acc);
        }
    __syncthreads(); // the staged records are read; the same memory takes the partial cells
    A* red = reinterpret_cast<A*>(smem);
    if (sub)
        for (int q = 0; q < C::NACC; q++)
            red[(q * kGridWarps + warp) * 32 + lane] = acc[q];
    __syncthreads();
    if (sub || br >= nbr)
        return;
    for (int w = first + 1; w < first + SPLIT; w++)
        for (int q = 0; q < C::NACC; q++)
            acc[q] += red[(q * kGridWarps + w) * 32 + lane];
    C::template store<1>(p, br * kBlk, bc * kBlk, acc);
}

// ---------------------------------------------------------------- separable kernels

template <typename R>
struct SepParams {
    int N, rows, pad, brn;
    int ld; // cells from one grid column to the next
    const uint32_t* off;
    const GridRec<R>* recs;
    const R* wts;      // per record (beam)
    const double* tab; // padded table (k_pad_table), or per-visibility kernels (k_exact_tables)
    int tw, zrow, K; // padded row length, position of the row of zeros
    void* grid;
    void* beam;
};

// Separable kernels on the FP64 tensor cores.  An entry adds the rank-one
// block kv (V ku)^T, so four entries are one 8 x 8 x 4 product: A holds the
// four v kernels at the block's rows, B the four u kernels at its columns
// times the visibility (one product for the real and one for the imaginary
// part), zeros where a footprint does not reach.  Two DMMA add four entries
// to all 64 cells; a lane looks up one tap of either axis per product.  The
// bound is instruction issue (about 5 warp instructions per entry and block)
// and the FP64 pipe (8 cycles); the shared-memory tile gridder it replaces
// spent about 85 warp instructions per entry and tile on decode and
// read-modify-write.  Calls, before and after: 4M visibilities on 8192^2
// (PSWF S = 4, compensated single precision) 2604 -> 1630 us; 100k on 2048^2
// in double 182 -> 159 us; 78k exact kernels with beam on 2160^2 (where the
// functor was evaluated per tap) 2016 -> 316 us.
// Products and sums are in double whatever the record's precision.  Entries
// with a weight, visibility or kernel that is not finite are added tap by
// tap instead, so that they reach their own footprint only.
template <typename R, typename G, bool EXACT, bool BEAM, bool STAB>
struct SepCore {
    using Params = SepParams<R>;
    using A = double;
    static constexpr int NACC = BEAM ? 6 : 4;
    static constexpr uint32_t kCta = BEAM ? 384 : 512;
    static constexpr int kMinBlocks = BEAM ? 3 : 5; // (4 blocks of 64 registers: 1460 us against 1421 on the 8192^2 call)
    struct Raw {
        GridRec<R> r;
        R w;
    };
    // ty, tx: table position of the entry's tap at the origin's row / column;
    // rc: row0 and col0 plus 512 (10 bits each), bit 20: exact, the mirrored
    // copy; bit 21: not finite
    struct alignas(16) StagedB {
        double vr, vi;
        int ty, tx;
        uint32_t vis, rc; // vis: exact, the visibility
        double w, unused;
    };
    struct alignas(16) StagedP {
        double vr, vi;
        int ty, tx;
        uint32_t vis, rc;
    };
    using Staged = std::conditional_t<BEAM, StagedB, StagedP>;
    static constexpr bool kOdd = true;
    static constexpr bool kWindows = true; // CTAs of more than kCta entries in several rounds
    // STAB: the padded table (at most kTab values) in shared memory.  The four
    // entries of a product read four runs of eight taps, up to eight lines of
    // L1 for a global load (which kept its data pipe 73 % busy on the 8192^2
    // call), about half as many passes over the banks.
    static constexpr int kTab = STAB ? 768 : 0;

    static __device__ __forceinline__ void load_table(const Params& p, double* s_tab)
    {
        if (STAB)
            for (int t = threadIdx.x; t < p.zrow + p.tw; t += blockDim.x)
                s_tab[t] = p.tab[t];
    }

    static __device__ __forceinline__ int bins(const Params& p) { return p.pad + 1; }
    static __device__ __forceinline__ Raw fetch(const Params& p, uint32_t i)
    {
        Raw w {};
        w.r = p.recs[i];
        if (BEAM)
            w.w = p.wts[i];
        return w;
    }
    static __device__ __forceinline__ Staged decode(const Params& p, const Raw& w, int r0, int c0)
    {
        Staged s;
        const uint32_t g = w.r.geom;
        const int row0 = int((g - uint32_t(r0)) << 22) >> 22, col0 = int((g - (uint32_t(c0) << 10)) << 12) >> 22;
        s.vr = double(w.r.vr);
        s.vi = double(w.r.vi);
        double chk = s.vr + s.vi;
        if constexpr (BEAM) {
            s.w = double(w.w);
            chk += s.w;
        }
        s.rc = uint32_t(row0 + 512) | (uint32_t(col0 + 512) << 10) | (((g >> 28) & 1u) << 20);
        // a kernel whose samples sum to zero is not finite in all its taps
        if (EXACT) {
            s.ty = -row0;
            s.tx = -col0;
            s.vis = w.r.koff;
            const double* t = p.tab + size_t(s.vis) * size_t(2 * p.K);
            chk += __ldg(t) + __ldg(t + p.K);
        } else {
            const int ky = int(w.r.koff & 0xffffu) * p.tw + 7, kx = int(w.r.koff >> 16) * p.tw + 7;
            s.ty = ky - row0;
            s.tx = kx - col0;
            s.vis = 0;
            chk += __ldg(p.tab + ky) + __ldg(p.tab + kx);
        }
        if (!(fabs(chk) <= 1.7976931348623157e308))
            s.rc |= 1u << 21;
        return s;
    }
    // an entry of zero weight for the block at (row, col)
    static __device__ __forceinline__ Staged dummy(const Params& p, int row, int col)
    {
        Staged z {};
        z.ty = EXACT ? -kBlk - row : p.zrow - row;
        z.tx = EXACT ? -kBlk - col : p.zrow - col;
        return z;
    }
    static __device__ __forceinline__ int row0_of(const Staged& s) { return int(s.rc & 1023u) - 512; }
    static __device__ __forceinline__ int col0_of(const Staged& s) { return int((s.rc >> 10) & 1023u) - 512; }
    static __device__ __forceinline__ bool odd(const Staged& s) { return (s.rc >> 21) & 1u; }
    static constexpr int kParts = 1;
    static __device__ __forceinline__ bool parts(const Params&) { return false; }
    template <int>
    static __device__ __forceinline__ unsigned reach(const Params& p, const Staged& s, int row, int col)
    {
        const int row0 = row0_of(s) - row, col0 = col0_of(s) - col;
        return row0 + p.K > 0 && row0 < kBlk && col0 + p.K > 0 && col0 < kBlk;
    }
    // the taps of either axis at the origin's row / column
    static __device__ __forceinline__ void taps(const Params& p, const double* stab, const Staged& s, int row, int col,
        double& a, double& b)
    {
        if (EXACT) {
            const int K = p.K;
            const int dr = s.ty + row, dc = s.tx + col;
            const bool back = (s.rc >> 20) & 1u;
            const double* t = p.tab + size_t(s.vis) * size_t(2 * K);
            a = unsigned(dr) < unsigned(K) ? __ldg(t + (back ? K - 1 - dr : dr)) : 0.0;
            b = unsigned(dc) < unsigned(K) ? __ldg(t + K + (back ? K - 1 - dc : dc)) : 0.0;
        } else if (STAB) {
            a = stab[s.ty + row];
            b = stab[s.tx + col];
        } else {
            a = __ldg(p.tab + s.ty + row);
            b = __ldg(p.tab + s.tx + col);
        }
    }
    // an entry that is not finite: its own footprint's cells only
    static __device__ __forceinline__ void add_odd(const Params& p, const double* stab, const Staged& s, int row, int col,
        A (&acc)[NACC])
    {
        const int lane = threadIdx.x & 31;
        for (int k = 0; k < 2; k++) {
            const int r = row + (lane >> 2), c = col + 2 * (lane & 3) + k;
            if (unsigned(r - row0_of(s)) < unsigned(p.K) && unsigned(c - col0_of(s)) < unsigned(p.K)) {
                double a, b;
                taps(p, stab, s, r, c, a, b);
                acc[k] += a * b * s.vr;
                acc[2 + k] += a * b * s.vi;
                if constexpr (BEAM)
                    acc[4 + k] += a * b * s.w;
            }
        }
    }
    static __device__ __forceinline__ void mma(double& c0, double& c1, double a, double b)
    {
        asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
            : "+d"(c0), "+d"(c1)
            : "d"(a), "d"(b));
    }
    template <int PARTS>
    static __device__ __forceinline__ void accumulate(const Params& p, const double* stab, const Staged* st,
        const uint16_t* list, int m, int row, int col, A (&acc)[NACC])
    {
        const int lane = threadIdx.x & 31;
        const int q = lane >> 2;
#pragma unroll 2
        for (int g = 0; g < m; g += 4) {
            const Staged& s = st[list[g + (lane & 3)]];
            double a, b;
            taps(p, stab, s, row + q, col + q, a, b);
            mma(acc[0], acc[1], a, b * s.vr);
            mma(acc[2], acc[3], a, b * s.vi);
            if constexpr (BEAM)
                mma(acc[4], acc[5], a, b * s.w);
        }
    }
    static __device__ __forceinline__ void store_zero(const Params& p, size_t i)
    {
        using G2 = typename Cplx<G>::T;
        static_cast<G2*>(p.grid)[i] = G2 {};
        if constexpr (BEAM)
            static_cast<G2*>(p.beam)[i] = G2 {};
    }
    // lane: row lane / 4, columns 2 (lane % 4) and the next
    template <int PARTS>
    static __device__ __forceinline__ void store(const Params& p, int r0, int c0, const A (&acc)[NACC])
    {
        using G2 = typename Cplx<G>::T;
        const int lane = threadIdx.x & 31;
        const int r = r0 + (lane >> 2);
        if (r >= p.rows)
            return;
#pragma unroll
        for (int k = 0; k < 2; k++) {
            const int c = c0 + 2 * (lane & 3) + k;
            if (c >= p.N)
                continue;
            const size_t i = size_t(c) * size_t(p.ld) + size_t(r);
            G2 v;
            v.x = G(acc[k]);
            v.y = G(acc[2 + k]);
            static_cast<G2*>(p.grid)[i] = v;
            if constexpr (BEAM) {
                G2 w;
                w.x = G(acc[4 + k]);
                w.y = G(0);
                static_cast<G2*>(p.beam)[i] = w;
            }
        }
    }
};

// ---------------------------------------------------------------- W-projection

template <typename R, typename T>
struct WprojParams {
    int N, rows, pad, brn;
    int ld; // cells from one grid column to the next
    const uint32_t* off;
    const GridRec<R>* recs;
    const R* wts;                     // per record (beam)
    const typename Cplx<T>::T* wk;    // expanded kernels: column j, row i at [koff + j K + i]
    const unsigned int* max_support; // largest support of the call's planes
    void* grid;
    void* beam;
};

// W-kernels: each lane keeps two cells of the block (row lane % 8, columns
// lane / 8 and that + 4; in two parts, two columns of its part) in registers
// and adds the entries one after the other: eight lanes read eight
// consecutive kernel values (rows of one column), so a warp's load touches the
// footprint's columns once each.  The
// kernel values of the next entries are in flight while one is added.  Sums
// (type A) are in double for FP64 and compensated FP32.
template <typename R, typename G, typename T, typename ACC, bool BEAM>
struct WprojCore {
    using Params = WprojParams<R, T>;
    using A = ACC;
    static constexpr int NACC = BEAM ? 8 : 4;
    // Most CTAs of the untruncated call of 1M visibilities on 4096^2 (support 16) in one go: 512 entries 2093 us, 960
    // 1743; 864 leave L1 a little more beside four CTAs an SM (132 KB of shared memory): 1726 with lists gathered for
    // one part, 960 1737.
    static constexpr uint32_t kCta = BEAM ? 720 : 864;
    static constexpr int kMinBlocks = BEAM ? 2 : 4; // (5 blocks of 48 registers spill: 472 us against 490 on the headline call)
    struct Raw {
        GridRec<R> r;
        R w;
    };
    struct alignas(16) StagedB {
        A vr, vi;
        int row0, col0;
        uint32_t koff;
        uint32_t kc; // K, and the sign bit when the kernel is conjugated
        A w, unused;
    };
    struct alignas(16) StagedP {
        A vr, vi;
        int row0, col0;
        uint32_t koff;
        uint32_t kc;
    };
    using Staged = std::conditional_t<BEAM, StagedB, StagedP>;

    static __device__ __forceinline__ int bins(const Params& p) { return int((2u * p.max_support[0] + 7u) / 8u) + 1; }
    static __device__ __forceinline__ Raw fetch(const Params& p, uint32_t i)
    {
        Raw w {};
        w.r = p.recs[i];
        if (BEAM)
            w.w = p.wts[i];
        return w;
    }
    static constexpr bool kWindows = false; // (the loop's registers: 206 -> 234 us on the double headline call)
    static constexpr bool kOdd = false; // (cells outside a footprint are not touched)
    static __device__ __forceinline__ bool odd(const Staged&) { return false; }
    static __device__ __forceinline__ void add_odd(const Params&, const double*, const Staged&, int, int, A (&)[NACC]) {}
    static constexpr int kTab = 0;
    static __device__ __forceinline__ void load_table(const Params&, double*) {}
    static __device__ __forceinline__ Staged decode(const Params&, const Raw& w, int r0, int c0)
    {
        Staged s;
        const uint32_t g = w.r.geom;
        s.row0 = int((g - uint32_t(r0)) << 22) >> 22;
        s.col0 = int((g - (uint32_t(c0) << 10)) << 12) >> 22;
        s.vr = A(w.r.vr);
        s.vi = A(w.r.vi);
        const int K = int(2u * ((g >> 20) & 127u) + 1u);
        s.koff = w.r.koff;
        s.kc = uint32_t(K) | ((g << 4) & 0x80000000u);
        if constexpr (BEAM)
            s.w = A(w.w);
        return s;
    }
    // an entry without taps
    static __device__ __forceinline__ Staged dummy(const Params&, int, int)
    {
        Staged z {};
        return z;
    }
    // a lane's first column, and from that to its second
    template <int PARTS>
    static __device__ __forceinline__ int lane_col(int lane)
    {
        return PARTS == 2 ? (lane >> 4) * 4 + ((lane >> 3) & 1) : lane >> 3;
    }
    // Small footprints in two parts, columns 0 to 3 and 4 to 7, each half of the
    // warp with an entry of its own: an entry of 5 x 5 cells reaches 11 of a
    // block's 64 on average, and two of three entries only one part.  Kernel on
    // the 1M-visibility 4096^2 call, one part and two: 196 and 179 us (truncated
    // to support 3 at most); untruncated support 3 216 and 196 (double 214 and
    // 205), 6 401 and 371 (397 and 387), 8 538 and 512 (528 and 537), 12 909 and
    // 879 to 968.
    static constexpr int kParts = 2;
    static __device__ __forceinline__ bool parts(const Params& p)
    {
        return p.max_support[0] <= (sizeof(T) == 4 ? 8u : 6u);
    }
    template <int PARTS>
    static __device__ __forceinline__ unsigned reach(const Params&, const Staged& s, int row, int col)
    {
        const int K = int(s.kc & 0xffffu), row0 = s.row0 - row, col0 = s.col0 - col, end = col0 + K;
        if (row0 + K <= 0 || row0 >= kBlk)
            return 0;
        if (PARTS == 1)
            return end > 0 && col0 < kBlk;
        return unsigned(end > 0 && col0 < kBlk / 2) | unsigned(end > kBlk / 2 && col0 < kBlk) << 1;
    }
    static __device__ __forceinline__ float flip(float x, uint32_t sign)
    {
        return __uint_as_float(__float_as_uint(x) ^ sign);
    }
    static __device__ __forceinline__ double flip(double x, uint32_t sign)
    {
        return __hiloint2double(int(uint32_t(__double2hiint(x)) ^ sign), __double2loint(x));
    }
    template <int PARTS>
    static __device__ __forceinline__ void accumulate(const Params& p, const double* stab, const Staged* st,
        const uint16_t* list, int m, int row, int col, A (&acc)[NACC])
    {
        using C2 = typename Cplx<T>::T;
        const int lane = threadIdx.x & 31;
        const int r = row + (lane & 7), c = col + lane_col<PARTS>(lane);
        constexpr int step = 4 / PARTS;
        const C2* __restrict__ wk = p.wk;
        if (PARTS == 2)
            list += (lane >> 4) * BlockList<PARTS>::kSize;
#pragma unroll 4
        for (int e = 0; e < m; e++) {
            const Staged s = st[list[e]];
            const int K = int(s.kc & 0xffffu);
            const uint32_t sign = s.kc & 0x80000000u;
            const int dr = r - s.row0, dc = c - s.col0;
            const bool in = unsigned(dr) < unsigned(K);
            const bool in0 = in && unsigned(dc) < unsigned(K), in1 = in && unsigned(dc + step) < unsigned(K);
            const uint32_t i = s.koff + uint32_t(dc * K + dr);
            C2 v[2];
            v[0].x = v[0].y = v[1].x = v[1].y = T(0);
            if (in0)
                v[0] = __ldg(wk + i);
            if (in1)
                v[1] = __ldg(wk + (i + uint32_t(step * K)));
#pragma unroll
            for (int k = 0; k < 2; k++) {
                if (k ? in1 : in0) {
                    const A kr = A(v[k].x), ki = A(flip(v[k].y, sign));
                    acc[2 * k] = fma(s.vr, kr, acc[2 * k]);
                    acc[2 * k] = fma(-s.vi, ki, acc[2 * k]);
                    acc[2 * k + 1] = fma(s.vr, ki, acc[2 * k + 1]);
                    acc[2 * k + 1] = fma(s.vi, kr, acc[2 * k + 1]);
                    if constexpr (BEAM) {
                        acc[4 + 2 * k] = fma(s.w, kr, acc[4 + 2 * k]);
                        acc[5 + 2 * k] = fma(s.w, ki, acc[5 + 2 * k]);
                    }
                }
            }
        }
    }
    static __device__ __forceinline__ void store_zero(const Params& p, size_t i)
    {
        using G2 = typename Cplx<G>::T;
        static_cast<G2*>(p.grid)[i] = G2 {};
        if constexpr (BEAM)
            static_cast<G2*>(p.beam)[i] = G2 {};
    }
    template <int PARTS>
    static __device__ __forceinline__ void store(const Params& p, int r0, int c0, const A (&acc)[NACC])
    {
        using G2 = typename Cplx<G>::T;
        const int lane = threadIdx.x & 31;
        const int r = r0 + (lane & 7);
        if (r >= p.rows)
            return;
#pragma unroll
        for (int k = 0; k < 2; k++) {
            const int c = c0 + lane_col<PARTS>(lane) + 4 / PARTS * k;
            if (c >= p.N)
                continue;
            const size_t i = size_t(c) * size_t(p.ld) + size_t(r);
            G2 v;
            v.x = G(acc[2 * k]);
            v.y = G(acc[2 * k + 1]);
            static_cast<G2*>(p.grid)[i] = v;
            if constexpr (BEAM) {
                G2 w;
                w.x = G(acc[4 + 2 * k]);
                w.y = G(acc[5 + 2 * k]);
                static_cast<G2*>(p.beam)[i] = w;
            }
        }
    }
};

} // namespace stpgpu
