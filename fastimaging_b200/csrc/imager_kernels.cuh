// Device kernels of the snapshot imager.
//
// Pipeline (one snapshot):
//   k_prepass      uvw -> pixel scaling, half-plane conversion, rint split,
//                  bounds check, uv shift, oversampled index  (gridder.h:369-504)
//   [W-proj]       plane boundaries/averages (k_wsel_*; a |w| sort, CUB, for
//                  what these do not take), FP64 W-kernels
//   k_bin_*, k_grid_blocks, k_grid_dense  binning and gridding
//                  (binning_kernels.cuh, gridder_kernels.cuh)
//   k_fft_axis, k_c2r_normalise  c2r, crop, 1/sum and gcf division of
//                  power-of-two grids (fft_kernels.cuh; fft.cpp:45-135,
//                  imager.h:97-150); other sizes cuFFT Z2D/C2R and k_normalise
#pragma once

#include "common.cuh"
#include "binning_kernels.cuh"

namespace stpgpu {

constexpr int GRID_THREADS = 256;

struct PrepassParams {
    int64_t n;
    const void* vis; // complex128 or complex64
    int vis_c64;
    const double* weights;
    const double* uv; // either uvw (n x 3, lambda) or uv (n x 2, pixels)
    int uv_is_pixels;
    double inv_px; // lambda -> pixel factor when uv_is_pixels == 0
    int N, conv_support, halfplane, shift_uv, kernel_exact, os;
    int keep_w;
    double* frac;      // 2n (exact mode only), may be null
    double* wsum_part; // per-block partial sums of good weights
    unsigned long long* ngood_part;
    double* absw_key; // n |w| (W-proj only), may be null
    double* wmax_part; // per block: the maximum and the sum of the finite |w| (W-proj), may be null
    uint32_t* iota;    // n identity permutation (W-proj), may be null
    unsigned int* ticket; // blocks done (zeroed before)
    double* total;        // results of the last block (finish_wsum)
    unsigned long long* ngood;
};

// Sum of block partials in a fixed order (one block of GRID_THREADS).  out[0]
// = 2 * sum (the half-plane doubling of gridder.h:423), out_n[0] = count;
// with mpart, out[1] = the largest finite |w| and out[2] = the sum of the
// finite |w|.
__device__ __forceinline__ void finish_wsum(const double* part, const unsigned long long* npart, const double* mpart, int nb,
    double* out, unsigned long long* out_n)
{
    __shared__ double s[GRID_THREADS], sm[GRID_THREADS], sa[GRID_THREADS];
    __shared__ unsigned long long sn[GRID_THREADS];
    double t = 0.0, m = 0.0, a = 0.0;
    unsigned long long c = 0;
    for (int k = threadIdx.x; k < nb; k += GRID_THREADS) {
        t += __ldcg(part + k);
        c += __ldcg(npart + k);
        if (mpart) {
            m = fmax(m, __ldcg(mpart + 2 * k));
            a += __ldcg(mpart + 2 * k + 1);
        }
    }
    s[threadIdx.x] = t;
    sn[threadIdx.x] = c;
    sm[threadIdx.x] = m;
    sa[threadIdx.x] = a;
    __syncthreads();
    for (int o = GRID_THREADS / 2; o > 0; o >>= 1) {
        if (int(threadIdx.x) < o) {
            s[threadIdx.x] += s[threadIdx.x + o];
            sn[threadIdx.x] += sn[threadIdx.x + o];
            sm[threadIdx.x] = fmax(sm[threadIdx.x], sm[threadIdx.x + o]);
            sa[threadIdx.x] += sa[threadIdx.x + o];
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        out[0] = s[0] * 2.0;
        out_n[0] = sn[0];
        if (mpart) {
            out[1] = sm[0];
            out[2] = sa[0];
        }
    }
}

// b.count: null with W-projection (the footprints are not known yet), else
// the entries are counted here.  The last block sums the blocks' partials.
template <typename R>
__global__ void __launch_bounds__(GRID_THREADS) k_prepass(PrepassParams p, Item<R>* items, BlockBins b)
{
    __shared__ double s_w[GRID_THREADS / 32];
    __shared__ unsigned long long s_n[GRID_THREADS / 32];
    __shared__ double s_m[GRID_THREADS / 32], s_a[GRID_THREADS / 32];
    double wgood = 0.0, wmax = 0.0, wabs = 0.0;
    unsigned long long ngood = 0;
    // a bounded number of blocks: the last one sums their partials
    for (int64_t i = int64_t(blockIdx.x) * GRID_THREADS + threadIdx.x; i < p.n; i += int64_t(gridDim.x) * GRID_THREADS) {
        double u, v, w = 0.0;
        if (p.uv_is_pixels) {
            u = p.uv[i];
            v = p.uv[p.n + i];
            if (p.keep_w)
                w = p.uv[2 * p.n + i];
        } else {
            u = p.uv[i] * p.inv_px;
            v = p.uv[p.n + i] * p.inv_px;
            w = p.uv[2 * p.n + i];
        }
        double vr, vi;
        if (p.vis_c64) {
            float2 t = reinterpret_cast<const float2*>(p.vis)[i];
            vr = t.x;
            vi = t.y;
        } else {
            double2 t = reinterpret_cast<const double2*>(p.vis)[i];
            vr = t.x;
            vi = t.y;
        }
        const double wt = p.weights[i];
        int good = 1;
        const int S = p.conv_support;
        if (p.halfplane) {
            if (v < 0.0) {
                if (v > -(S + 1))
                    good = 2;
                u *= -1;
                v *= -1;
                w *= -1;
                vi = -vi;
            } else if (v < (S + 1)) {
                good = 2;
            }
        }
        const int half = p.N / 2;
        bool finite = isfinite(u) && isfinite(v);
        double ru = rint(u), rv = rint(v);
        // int(rint(x)) with the out-of-range behaviour of x86 (INT_MIN) kept
        // for the bounds check: such centres are always out of bounds.
        long long vx = (finite && fabs(ru) < 1.0e9) ? (long long)ru : (long long)INT32_MIN;
        long long vy = (finite && fabs(rv) < 1.0e9) ? (long long)rv : (long long)INT32_MIN;
        double fx = u - double(vx), fy = v - double(vy);
        long long kx = vx + half, ky = vy + half;
        if (!finite || (kx - S) <= 0 || (ky - S) <= 0 || (kx + S) >= p.N || (ky + S) >= p.N)
            good = 0;
        if (p.shift_uv) {
            kx = kx < half ? kx + half : kx - half;
            ky = ky < half ? ky + half : ky - half;
        }
        int cpx = 0, cpy = 0;
        if (!p.kernel_exact) {
            const int rmax = p.os / 2;
            int ox = int(rint(fx * p.os)), oy = int(rint(fy * p.os));
            ox = ox > rmax ? rmax : (ox < -rmax ? -rmax : ox);
            oy = oy > rmax ? rmax : (oy < -rmax ? -rmax : oy);
            cpx = ox + rmax;
            cpy = oy + rmax;
        }
        if (p.frac) {
            p.frac[i] = fx;
            p.frac[p.n + i] = fy;
        }
        if (p.absw_key)
            p.absw_key[i] = fabs(w);
        if (fabs(w) <= 1.7976931348623157e308) { // finite
            wmax = fmax(wmax, fabs(w));
            wabs += fabs(w);
        }
        if (p.iota)
            p.iota[i] = uint32_t(i);
        Item<R> it;
        it.vr = R(vr);
        it.vi = R(vi);
        it.w = R(wt);
        it.gcx = good ? int32_t(kx) : 0;
        it.gcy = good ? int32_t(ky) : 0;
        it.cpx = int16_t(cpx);
        it.cpy = int16_t(cpy);
        it.plane = 0;
        it.good = uint8_t(good);
        it.flags = uint8_t((w < 0.0 ? 1 : 0) | (-w < 0.0 ? 2 : 0));
        items[i] = it;
        if (good) {
            wgood += wt;
            ngood++;
            if (b.count)
                count_entries(b, it, i, b.support);
        }
    }
    // deterministic block partial sums
    for (int o = 16; o > 0; o >>= 1) {
        wgood += __shfl_down_sync(0xffffffffu, wgood, o);
        ngood += __shfl_down_sync(0xffffffffu, ngood, o);
        wmax = fmax(wmax, __shfl_down_sync(0xffffffffu, wmax, o));
        wabs += __shfl_down_sync(0xffffffffu, wabs, o);
    }
    if ((threadIdx.x & 31) == 0) {
        s_w[threadIdx.x >> 5] = wgood;
        s_n[threadIdx.x >> 5] = ngood;
        s_m[threadIdx.x >> 5] = wmax;
        s_a[threadIdx.x >> 5] = wabs;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0, m = 0.0, a = 0.0;
        unsigned long long c = 0;
        for (int k = 0; k < int(blockDim.x >> 5); k++) {
            t += s_w[k];
            c += s_n[k];
            m = fmax(m, s_m[k]);
            a += s_a[k];
        }
        p.wsum_part[blockIdx.x] = t;
        p.ngood_part[blockIdx.x] = c;
        if (p.wmax_part) {
            p.wmax_part[2 * blockIdx.x] = m;
            p.wmax_part[2 * blockIdx.x + 1] = a;
        }
    }
    if (last_block(p.ticket))
        finish_wsum(p.wsum_part, p.ngood_part, p.wmax_part, int(gridDim.x), p.total, p.ngood);
}

// Sort keys of |w| for the W-plane order, 24 bits, monotone in |w| (|a| <=
// |b| implies key(a) <= key(b)), so that a stable sort of the keys followed
// by k_fix_runs (runs of equal keys re-sorted by the full |w| bits, NaN after
// every number) gives the order of the IEEE bits of |w|.  With x = |w| /
// wmax (wmax = total[1], the largest finite |w|), two encodings, chosen by
// how far the mean |w| (total[2] / n) sits below wmax so that runs of equal
// keys stay short:
//  * spread |w| (mean >= wmax / 16): floor(sqrt(x) (2^24 - 2)), resolution
//    2^-24 in sqrt(x) (about 8 % of the headline snapshot's keys in runs);
//  * |w| concentrated far below wmax: x rounded down to single precision and
//    raised to at least 2^-31, key = (bits(x) - bits(2^-31)) >> 4 (the 32
//    exponents from 2^-31 to 1 and 19 mantissa bits: relative resolution
//    2^-19 at every scale).
// Non-finite |w| (NaN included) take 2^24 - 1, above every finite key.
struct WKey {
    double wmax, r;
    bool spread;
    __device__ WKey(const double* total, int64_t n)
    {
        wmax = total[1];
        r = wmax > 0.0 ? 1.0 / wmax : 0.0;
        spread = wmax > 0.0 && total[2] >= wmax * 0.0625 * double(n);
    }
    __device__ __forceinline__ uint32_t operator()(double a) const
    {
        uint32_t k = 0xFFFFFFu;
        if (a <= wmax) {
            if (spread) {
                const double q = __dsqrt_rn(a * r) * 16777214.0;
                k = q < 16777214.0 ? uint32_t(q) : 16777214u;
            } else {
                const float x = fmaxf(__double2float_rd(a * r), 0x1p-31f);
                k = (__float_as_uint(x) - 0x30000000u) >> 4;
            }
        }
        return k;
    }
};

__global__ void k_wkey24(const double* __restrict__ absw, int64_t n, const double* total, uint32_t* __restrict__ key)
{
    const WKey kf(total, n);
    for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x)
        key[i] = kf(absw[i]);
}

// Zeroes up to four ranges of 32-bit words (one launch instead of several
// memset nodes in a captured call).
struct ZeroRanges {
    uint32_t* p[4];
    int64_t n[4];
};
__global__ void k_zero_ranges(ZeroRanges z)
{
    const int64_t t = int64_t(blockIdx.x) * blockDim.x + threadIdx.x, st = int64_t(gridDim.x) * blockDim.x;
#pragma unroll
    for (int r = 0; r < 4; r++)
        if (z.p[r])
            for (int64_t i = t; i < z.n[r]; i += st)
                z.p[r][i] = 0;
}

// Exclusive scan of n counts into off[0..n] (single block of 1024 threads,
// n up to a few hundred thousand).  off[n] = total.  Each thread first
// loads 16 elements (16 coalesced rows of 1024), then the rows are scanned
// in order with warp shuffles and one shared-memory step per row.
__device__ __forceinline__ uint32_t scan_block_1024(const uint32_t* cnt, uint32_t* off, int n)
{
    __shared__ uint32_t wsum[32];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    uint32_t carry = 0;
    for (int base = 0; base < n; base += 1024 * 16) {
        uint32_t v[16];
#pragma unroll
        for (int j = 0; j < 16; j++) {
            const int idx = base + j * 1024 + tid;
            v[j] = idx < n ? cnt[idx] : 0u;
        }
#pragma unroll
        for (int j = 0; j < 16; j++) {
            if (base + j * 1024 >= n)
                break;
            uint32_t x = v[j];
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
                if (lane >= o)
                    x += y;
            }
            if (lane == 31)
                wsum[warp] = x;
            __syncthreads();
            if (warp == 0) {
                uint32_t t = wsum[lane];
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const uint32_t y = __shfl_up_sync(0xffffffffu, t, o);
                    if (lane >= o)
                        t += y;
                }
                wsum[lane] = t;
            }
            __syncthreads();
            const int idx = base + j * 1024 + tid;
            if (idx < n)
                off[idx] = carry + (warp ? wsum[warp - 1] : 0u) + x - v[j];
            carry += wsum[31];
            __syncthreads();
        }
    }
    if (tid == 0)
        off[n] = carry;
    return carry;
}

// One such scan per block: row blockIdx.x of cnt and off (row stride
// `stride`); the totals also go to tot[row].
__global__ void __launch_bounds__(1024) k_scan_rows(const uint32_t* cnt, uint32_t* off, int n, int stride, uint32_t* tot)
{
    const uint32_t t = scan_block_1024(cnt + int64_t(blockIdx.x) * stride, off + int64_t(blockIdx.x) * stride, n);
    if (threadIdx.x == 0)
        tot[blockIdx.x] = t;
}

template <typename R>
struct Cplx;
template <>
struct Cplx<double> {
    using T = double2;
};
template <>
struct Cplx<float> {
    using T = float2;
};

// ---------------------------------------------------------------- kernel tables

// make_1D_kernel for every oversampled offset (populate_kernel_cache,
// gridder.h:73-105): out[cs][K], normalised by accu (two accumulators).
__global__ void k_kernel_table(int kf, double trunc, int support, int os, double* out)
{
    const int half = os / 2;
    const int cs = half * 2 + 1;
    const int K = 2 * support + 1;
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= cs)
        return;
    const double offset = (double(c) - half) / os;
    double a1 = 0.0, a2 = 0.0;
    for (int i = 0; i < K; i++) {
        double d = (double(i) - support) / 1;
        double v = kernel_value(kf, trunc, d - offset);
        out[c * K + i] = v;
        if (i & 1)
            a2 += v;
        else
            a1 += v;
    }
    const double s = a1 + a2;
    for (int i = 0; i < K; i++)
        out[c * K + i] = out[c * K + i] / s;
}

// ImgDomKernel (conv_func.h:351-412).  Analytic: gcf((i - c)/c).  Otherwise
// the real part of the R2HC DFT of the normalised, wrapped 1-D kernel,
// mirrored about the centre.  The kernel is exactly zero beyond `trunc`, so
// the DFT is a short cosine sum, evaluated with exact argument reduction.
__global__ void k_imgdom_kernel(int kf, double trunc, int n, int analytic, double ksum_inv, int dmax, double* out)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n)
        return;
    const int centre = n / 2;
    if (analytic) {
        out[i] = gcf_value(kf, (double(i) - centre) / centre);
        return;
    }
    // aa[n/2 + m] = r_m (m < n/2), aa[n/2 - m] = r_m (1 <= m <= n/2)
    int m = i >= centre ? i - centre : centre - i;
    double r = 0.0;
    // arr[j] = k1(j) (j < n/2), k1(j - n) (j >= n/2); r_m = sum_j arr[j] cos(2 pi j m / n)
    for (int d = -dmax; d <= dmax; d++) {
        if (d < -centre || d >= n - centre)
            continue;
        double kv = kernel_value(kf, trunc, double(d));
        if (kv == 0.0)
            continue;
        kv = kv * ksum_inv;
        long long jm = (long long)(d < 0 ? d + n : d) * m % n;
        r += kv * cospi(2.0 * double(jm) / double(n));
    }
    out[i] = r;
}

// The scalars a call reads back: sampling-grid total, good visibilities,
// binned entries, error flags and the largest plane support.  One warp
// writes them straight into page-locked host memory through its device
// address; the normalisation, a call's last kernel, does it in its first
// block (out non-null), so that they cost no launch of their own.
struct ScalarPack {
    double total;
    unsigned long long ngood;
    uint32_t nitems;
    unsigned int err;
    int max_support;
    int pad;
};

struct PackArgs {
    const double* total;
    const unsigned long long* ngood;
    const uint32_t* nitems;
    const unsigned int* err;
    const int* sup;
    int nsup;
    ScalarPack* out;
};

__device__ __forceinline__ void pack_scalars(const PackArgs& k)
{
    int m = 0;
    for (int i = threadIdx.x; i < k.nsup; i += 32)
        m = max(m, k.sup[i]);
    for (int o = 16; o > 0; o >>= 1)
        m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
    if (threadIdx.x == 0) {
        k.out->total = *k.total;
        k.out->ngood = *k.ngood;
        k.out->nitems = *k.nitems;
        k.out->err = *k.err;
        k.out->max_support = m;
        k.out->pad = 0;
    }
}

// ---------------------------------------------------------------- normalise

// normalise_image_beam_result_1D, non-FFTSHIFT branch (imager.h:97-150):
// crop the padded image keeping the unshifted quadrant layout, multiply by
// 1/sum and divide by gcf[ii]*gcf[jj].  blockIdx.y = output column; the
// factor 1/sum is read from the device (0 when the sampling total is 0).
template <typename RI, typename RO>
__global__ void __launch_bounds__(256) k_normalise(const RI* __restrict__ img, int padded, int image_size,
    const double* total, const double* __restrict__ ginv, int corr, RO* __restrict__ out, PackArgs pk)
{
    if (pk.out && blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x < 32)
        pack_scalars(pk);
    const int j = blockIdx.y;
    const double tot = total[0];
    const double nf = tot > 0.0 ? 1.0 / tot : 0.0;
    const int hp = padded / 2, hs = image_size / 2;
    const int oj = j < hs ? j : padded + j - image_size;
    const int jj = j < hs ? j + hp : hp + j - image_size;
    // value * (1/sum) / (gcf[ii] * gcf[jj]) as value * (nf * 1/gcf[jj]) * 1/gcf[ii]
    const double fj = corr ? nf * ginv[jj] : nf;
    const RI* src = img + size_t(oj) * padded;
    RO* dst = out + size_t(j) * image_size;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < image_size; i += gridDim.x * blockDim.x) {
        const int oi = i < hs ? i : padded - hs + (i - hs);
        const int ii = i < hs ? hp + i : hp - hs + (i - hs);
        const double v = double(src[oi]) * fj;
        dst[i] = RO(corr ? v * ginv[ii] : v);
    }
}

// Same pass, four rows per thread with 16-byte loads and stores, for
// image_size % 8 == 0 and padded % 4 == 0 (each group of four rows then lies
// inside one crop segment and is 16-byte aligned).  blockIdx.y = a group of
// kNormCols output columns: a thread keeps its rows' 1/gcf for all of them
// and has their loads in flight together (one short block per column spent
// more time in block scheduling than in the copy).
constexpr int kNormCols = 8;
template <typename RI, typename RO>
__global__ void __launch_bounds__(256) k_normalise4(const RI* __restrict__ img, int padded, int image_size,
    const double* total, const double* __restrict__ ginv, int corr, RO* __restrict__ out, PackArgs pk)
{
    if (pk.out && blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x < 32)
        pack_scalars(pk);
    const double tot = total[0];
    const double nf = tot > 0.0 ? 1.0 / tot : 0.0;
    const int hp = padded / 2, hs = image_size / 2;
    const int groups = image_size / 4;
    for (int g = blockIdx.x * blockDim.x + threadIdx.x; g < groups; g += gridDim.x * blockDim.x) {
        const int i = g * 4;
        const int oi = i < hs ? i : padded - hs + (i - hs);
        const int ii = i < hs ? hp + i : hp - hs + (i - hs);
        double gi[4];
#pragma unroll
        for (int k = 0; k < 4; k++)
            gi[k] = corr ? ginv[ii + k] : 1.0;
        RI x[kNormCols][4];
#pragma unroll
        for (int c = 0; c < kNormCols; c++) {
            const int j = blockIdx.y * kNormCols + c;
            if (j >= image_size)
                break;
            const int oj = j < hs ? j : padded + j - image_size;
            const RI* src = img + size_t(oj) * padded + oi;
            if constexpr (sizeof(RI) == 4) {
                const float4 q = *reinterpret_cast<const float4*>(src);
                x[c][0] = q.x;
                x[c][1] = q.y;
                x[c][2] = q.z;
                x[c][3] = q.w;
            } else {
                const double2 a = *reinterpret_cast<const double2*>(src);
                const double2 b = *reinterpret_cast<const double2*>(src + 2);
                x[c][0] = a.x;
                x[c][1] = a.y;
                x[c][2] = b.x;
                x[c][3] = b.y;
            }
        }
#pragma unroll
        for (int c = 0; c < kNormCols; c++) {
            const int j = blockIdx.y * kNormCols + c;
            if (j >= image_size)
                break;
            const int jj = j < hs ? j + hp : hp + j - image_size;
            const double fj = corr ? nf * ginv[jj] : nf;
            double v[4];
#pragma unroll
            for (int k = 0; k < 4; k++) {
                v[k] = double(x[c][k]) * fj;
                if (corr)
                    v[k] *= gi[k];
            }
            RO* dst = out + size_t(j) * image_size + i;
            if constexpr (sizeof(RO) == 4) {
                *reinterpret_cast<float4*>(dst) = make_float4(float(v[0]), float(v[1]), float(v[2]), float(v[3]));
            } else {
                *reinterpret_cast<double2*>(dst) = make_double2(v[0], v[1]);
                *reinterpret_cast<double2*>(dst + 2) = make_double2(v[2], v[3]);
            }
        }
    }
}

__global__ void k_reciprocal(const double* in, double* out, int n)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n)
        out[i] = 1.0 / in[i];
}

// ---------------------------------------------------------------- W-projection

// Plane boundaries (average_w_planes, gridder.cpp:68-146) from the |w|-sorted
// order: cgood[k] = number of good visibilities among sorted[0..k).  A plane
// ends behind its last good visibility, so the boundaries are a chain with
// one look-up per plane in goodpos (sorted position of every good
// visibility), which all blocks fill and the last one then follows.  (A
// binary search in cgood per plane: 199 us for 64 planes of 333k.)
__global__ void __launch_bounds__(256) k_wplanes(const uint32_t* __restrict__ cgood, int64_t n, int P, uint32_t* goodpos,
    unsigned int* ticket, int64_t* first, int64_t* last)
{
    for (int64_t k = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; k < n; k += int64_t(gridDim.x) * blockDim.x) {
        const uint32_t g = cgood[k];
        if (cgood[k + 1] != g)
            goodpos[g] = uint32_t(k);
    }
    if (!last_block(ticket) || threadIdx.x != 0)
        return;
    const uint64_t G = cgood[n];
    uint64_t begin = 0, before = 0; // good visibilities before `begin`
    for (int idx = 0; idx < P; idx++) {
        const uint64_t plane_size = uint64_t(ceil(double(G - begin) / (P - idx)));
        const uint64_t remaining = G - before;
        uint64_t end = begin;
        if (plane_size > remaining) {
            end = uint64_t(n);
            before = G;
        } else if (plane_size > 0) {
            before += plane_size;
            end = uint64_t(__ldcg(goodpos + before - 1)) + 1;
        }
        first[idx] = int64_t(begin);
        last[idx] = int64_t(end);
        begin = end;
    }
}

// One block per plane: plane w = mean |w| over good visibilities (or the
// median rule), in the plane's sorted range.
__global__ void k_wplane_values(const uint32_t* cgood, const double* absw_sorted, const uint8_t* good_sorted,
    const int64_t* first, const int64_t* last, int64_t n, int P, int median, double* w_avg)
{
    const int p = blockIdx.x;
    const int64_t b = first[p], e = last[p];
    __shared__ double s[256];
    if (!median) {
        double t = 0.0;
        for (int64_t k = b + threadIdx.x; k < e; k += blockDim.x)
            if (good_sorted[k])
                t += absw_sorted[k];
        s[threadIdx.x] = t;
        __syncthreads();
        for (int o = blockDim.x / 2; o > 0; o >>= 1) {
            if (threadIdx.x < o)
                s[threadIdx.x] += s[threadIdx.x + o];
            __syncthreads();
        }
        if (threadIdx.x == 0) {
            uint64_t cnt = uint64_t(cgood[e]) - uint64_t(cgood[b]);
            w_avg[p] = cnt > 0 ? s[0] / double(cnt) : 0.0;
        }
    } else if (threadIdx.x == 0) {
        // median variant (gridder.cpp:79-118)
        const uint64_t G = cgood[n];
        uint64_t plane_size = uint64_t(ceil(double(G - uint64_t(b)) / (P - p)));
        uint64_t middle = plane_size / 2;
        if (uint64_t(b) + plane_size > G)
            middle = (G - uint64_t(b)) / 2;
        uint64_t counter = uint64_t(cgood[e]) - uint64_t(cgood[b]);
        if (counter == 0) {
            w_avg[p] = 0.0;
            return;
        }
        // idx_mid: position of the (middle)-th good from b
        uint64_t target = uint64_t(cgood[b]) + middle; // cgood[k] == target and good[k]
        int64_t lo = b, hi = e;
        while (lo < hi) {
            int64_t mid = (lo + hi) / 2;
            if (uint64_t(cgood[mid + 1]) > target)
                hi = mid;
            else
                lo = mid + 1;
        }
        int64_t idx_mid = lo;
        if ((plane_size % 2) == 0 && idx_mid > 0)
            w_avg[p] = (absw_sorted[idx_mid - 1] + absw_sorted[idx_mid]) / 2.0;
        else
            w_avg[p] = absw_sorted[idx_mid];
    }
}

// Mean |w| per plane in two deterministic steps: block b sums the good |w|
// of its slice [b*chunk, (b+1)*chunk) of the sorted array separately for
// every plane the slice meets (partial[p][b]); then one block per plane adds
// its partials in block order.
__global__ void __launch_bounds__(256) k_wplane_partial(const double* __restrict__ absw_sorted,
    const uint8_t* __restrict__ good_sorted, const int64_t* first, const int64_t* last, int64_t n, int P,
    int64_t chunk, int nblk, double* partial)
{
    __shared__ double red[256];
    const int64_t a = int64_t(blockIdx.x) * chunk;
    const int64_t b = min(n, a + chunk);
    if (a >= b)
        return;
    int p = 0;
    {
        int lo = 0, hi = P - 1; // last plane with first <= a
        while (lo < hi) {
            const int mid = (lo + hi + 1) / 2;
            if (first[mid] <= a)
                lo = mid;
            else
                hi = mid - 1;
        }
        p = lo;
    }
    for (; p < P && first[p] < b; p++) {
        const int64_t s0 = max(a, first[p]), s1 = min(b, last[p]);
        double t = 0.0;
#pragma unroll 2
        for (int64_t k = s0 + threadIdx.x; k < s1; k += blockDim.x)
            if (good_sorted[k])
                t += absw_sorted[k];
        red[threadIdx.x] = t;
        __syncthreads();
        for (int o = blockDim.x / 2; o > 0; o >>= 1) {
            if (threadIdx.x < o)
                red[threadIdx.x] += red[threadIdx.x + o];
            __syncthreads();
        }
        if (threadIdx.x == 0)
            partial[int64_t(p) * nblk + blockIdx.x] = red[0];
        __syncthreads();
    }
}

__global__ void __launch_bounds__(256) k_wplane_finish(const double* partial, const uint32_t* cgood,
    const int64_t* first, const int64_t* last, int64_t chunk, int nblk, double* w_avg)
{
    __shared__ double red[256];
    const int p = blockIdx.x;
    const int64_t f = first[p], l = last[p];
    double t = 0.0;
    if (l > f) {
        const int b0 = int(f / chunk), b1 = int((l - 1) / chunk);
        for (int bb = b0 + int(threadIdx.x); bb <= b1; bb += blockDim.x)
            t += partial[int64_t(p) * nblk + bb];
    }
    red[threadIdx.x] = t;
    __syncthreads();
    for (int o = blockDim.x / 2; o > 0; o >>= 1) {
        if (threadIdx.x < o)
            red[threadIdx.x] += red[threadIdx.x + o];
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        const uint64_t cnt = uint64_t(cgood[l]) - uint64_t(cgood[f]);
        w_avg[p] = cnt > 0 ? red[0] / double(cnt) : 0.0;
    }
}

template <typename R>
__global__ void k_gather_good(const uint32_t* perm, const Item<R>* items, const double* absw, int64_t n,
    uint8_t* good_sorted, uint32_t* gflag, double* absw_sorted, Item<R>* items_sorted)
{
    const int64_t k = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (k >= n)
        return;
    const uint32_t i = perm[k];
    const Item<R> it = items[i];
    uint8_t g = it.good != 0;
    good_sorted[k] = g;
    gflag[k] = g;
    if (absw_sorted)
        absw_sorted[k] = absw[i];
    if (items_sorted)
        items_sorted[k] = it; // binning and gridding read the items in |w| order
}

// ---------------------------------------------------------------- W-planes without the |w| sort
//
// The reference's W-planes (gridder.cpp:68-146) take equal counts of the
// |w|-sorted visibilities.  When every visibility is good, plane p holds the
// sorted ranks [G_p, G_p+1) with G_0 = 0, G_p+1 = G_p + ceil((n - G_p) / (P -
// p)), so an item's plane follows from how many plane-start items precede
// it in the sort order ((|w| bits, input index), the stable order).  Those
// P - 1 items are found without sorting: a histogram of the 24-bit keys'
// top 12 to 16 bits places each start rank in a bin and at a rank within it
// (k_wsel_hist and, in its last block, wsel_plan); the members of those bins are collected
// (k_wsel_collect) and each start item is the member of its bin with the
// wanted rank under the exact order (k_wsel_resolve: every member counts the
// members before it).  k_wsel_classify then gives every item its plane (a
// binary search over the start items) and sums |w| per plane exactly, in
// 64-bit fixed point relative to the plane's smallest |w| (so the sums do
// not depend on the order of the additions); its last block forms the means
// and plane starts.  Items not all good, non-finite |w|, more than WSEL_MAXP
// planes or a start bin of more than WSEL_CAP members set bit 16 of the
// error word: the host then runs the sorting path.
// Bins: a power of two near n / 8 (about ten members in a start bin; small
// calls plan over fewer bins), key24 >> (24 - blog).
constexpr int WSEL_MIN_LOG = 12, WSEL_MAX_LOG = 16;
constexpr int WSEL_BINS = 1 << WSEL_MAX_LOG;
constexpr int WSEL_CAP = 2048;  // members of a start item's bin that k_wsel_resolve holds
constexpr int WSEL_MAXP = 1024; // planes

struct WselState {
    // zeroed before the pass
    uint32_t hist[WSEL_BINS];
    uint32_t cursor[WSEL_MAXP];
    uint32_t tickets[2];
    unsigned long long sum[WSEL_MAXP];
    // written by wsel_plan / k_wsel_resolve
    int32_t binmap[WSEL_BINS];      // list of a start bin, -1 otherwise
    uint32_t list_off[WSEL_MAXP + 1];
    uint32_t list_cnt[WSEL_MAXP];
    int32_t start_list[WSEL_MAXP];  // per plane p >= 1: its start item's list
    uint32_t start_rank[WSEL_MAXP]; // and rank within the list's bin
    uint32_t start_bin[WSEL_MAXP];
    unsigned long long start_bits[WSEL_MAXP]; // the start item: |w| bits, input index
    uint32_t start_idx[WSEL_MAXP];
    int64_t G[WSEL_MAXP + 1];
    int valid;
};
constexpr size_t kWselZeroWords = (sizeof(uint32_t) * (WSEL_MAXP + 2) + sizeof(unsigned long long) * WSEL_MAXP) / 4; // beside hist

// Exclusive scan over the 1024 threads of a block of the values v; *total =
// their sum.
__device__ __forceinline__ uint32_t wsel_block_scan(uint32_t v, uint32_t* total)
{
    __shared__ uint32_t wsum[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t x = v;
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o)
            x += y;
    }
    if (lane == 31)
        wsum[warp] = x;
    __syncthreads();
    if (warp == 0) {
        uint32_t w = wsum[lane];
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o)
                w += y;
        }
        wsum[lane] = w; // inclusive over the warps
    }
    __syncthreads();
    const uint32_t r = x - v + (warp ? wsum[warp - 1] : 0u);
    *total = wsum[31];
    __syncthreads();
    return r;
}

// One block of 1024 threads.  The plane starts have a closed form: with q =
// n / P and r = n % P, ceil((n - G_p) / (P - p)) = q + [p < r], so G_p = p q +
// min(p, r).  A block scan of the totals of 1024 chunks of bins locates
// each start rank's chunk, and the plane's thread walks the chunk's bins to
// the bin and the rank within it.  The start bins become lists in plane order.
__device__ __forceinline__ void wsel_plan(WselState* ws, int blog, int64_t n, int P, const unsigned long long* ngood,
    unsigned int* err)
{
    const int per = 1 << (blog - 10); // bins per chunk, 4 to 64
    __shared__ uint32_t chunk[1025]; // prefix at each thread's first bin
    const int tid = threadIdx.x;
    const bool ok0 = ngood[0] == (unsigned long long)n && P >= 1 && P <= WSEL_MAXP;
    // totals of the 1024 chunks: four bins a lane, so that a load covers whole
    // lines (a thread reading its own chunk touches 32 lines per load)
    {
        const int lane = tid & 31, warp = tid >> 5, lanes = per / 4; // lanes per chunk
        const uint4* c4 = reinterpret_cast<const uint4*>(ws->hist) + warp * (32 * lanes);
#pragma unroll 8
        for (int c = 0; c < lanes; c++) {
            const uint4 v = __ldcg(c4 + c * 32 + lane);
            uint32_t t = v.x + v.y + v.z + v.w;
            for (int o = lanes / 2; o > 0; o >>= 1)
                t += __shfl_xor_sync(0xffffffffu, t, o);
            if ((lane & (lanes - 1)) == 0)
                chunk[warp * 32 + (c * 32 + lane) / lanes] = t;
        }
        __syncthreads();
    }
    const uint32_t t = chunk[tid];
    uint32_t total = 0;
    const uint32_t excl = wsel_block_scan(t, &total);
    chunk[tid] = excl;
    if (tid == 0)
        chunk[1024] = total;
    const int64_t qn = P >= 1 ? n / P : 0, rn = P >= 1 ? n % P : 0;
    auto G = [&](int p) { return int64_t(p) * qn + (int64_t(p) < rn ? int64_t(p) : rn); };
    if (ok0)
        for (int p = tid; p <= P; p += blockDim.x)
            ws->G[p] = G(p);
    __syncthreads();
    // each plane's start item: its bin (the last b whose prefix is <= G_p), the
    // rank within it and the bin's size.  One warp per plane, two bins of the
    // start's chunk a lane: a thread walking the chunk alone waits for up to
    // 16 loads in turn (19 us of a 5k-visibility call)
    __shared__ uint32_t ssize[1024], srank[1024], sbin[1024];
    const int lane = tid & 31;
    for (int p = tid >> 5; p < 1024; p += 32) {
        if (!(ok0 && p >= 1 && p < P && G(p) < n))
            continue;
        const uint32_t gp = uint32_t(G(p));
        int lo = 0, hi = 1023;
        while (lo < hi) {
            const int mid = (lo + hi + 1) / 2;
            if (chunk[mid] <= gp)
                lo = mid;
            else
                hi = mid - 1;
        }
        const uint2 v = 2 * lane < per ? __ldcg(reinterpret_cast<const uint2*>(ws->hist + per * lo) + lane) : make_uint2(0u, 0u);
        uint32_t x = v.x + v.y;
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o)
                x += y;
        }
        const uint32_t end = chunk[lo] + x; // entries up to the lane's second bin
        const int at = __ffs(int(__ballot_sync(0xffffffffu, end > gp))) - 1;
        if (lane == at) {
            const uint32_t first = end - v.x - v.y; // before the lane's first bin
            const bool second = first + v.x <= gp;
            sbin[p] = uint32_t(per * lo + 2 * lane) + (second ? 1u : 0u);
            srank[p] = gp - (second ? first + v.x : first);
            ssize[p] = second ? v.y : v.x;
        }
    }
    __syncthreads();
    const int p = tid;
    const bool has = ok0 && p >= 1 && p < P && G(p) < n;
    const uint32_t bin = has ? sbin[p] : 0u, m = has ? ssize[p] : 0u;
    if (has) {
        ws->start_bin[p] = bin;
        ws->start_rank[p] = srank[p];
    }
    __shared__ int bad;
    if (!has)
        sbin[tid] = 0;
    if (tid == 0)
        bad = !ok0;
    __syncthreads();
    // a start bin opens a list unless the previous plane's start is in it
    const bool opens = has && !(p >= 2 && G(p - 1) < n && sbin[p - 1] == bin);
    if (opens && m > uint32_t(WSEL_CAP))
        bad = 1;
    uint32_t nlist = 0, noff = 0;
    const uint32_t li = wsel_block_scan(opens ? 1u : 0u, &nlist);
    const uint32_t off = wsel_block_scan(opens ? m : 0u, &noff);
    __shared__ uint32_t slist[1024];
    slist[tid] = opens ? li : 0u;
    __syncthreads();
    if (bad) {
        if (tid == 0) {
            ws->valid = 0;
            atomicOr(err, 16u);
        }
        return;
    }
    if (opens) {
        ws->binmap[bin] = int32_t(li);
        ws->list_off[li] = off;
        ws->list_cnt[li] = m;
    }
    if (p >= 1 && p < P) {
        // the list of this plane's start: that of the last plane up to p that
        // opened one (planes after the items run out have none)
        int32_t l = -1;
        if (has) {
            int q = p;
            while (q >= 2 && G(q - 1) < n && sbin[q - 1] == bin)
                q--;
            l = int32_t(slist[q]);
        }
        ws->start_list[p] = l;
    }
    if (tid == 0) {
        ws->list_off[nlist] = noff;
        ws->valid = 1;
    }
}

// Histogram of the 24-bit keys (those of k_wkey24, formed here and again in
// k_wsel_collect from |w|), then the plan by the last block.
__global__ void __launch_bounds__(1024) k_wsel_hist(const double* __restrict__ absw, int64_t n, const double* total,
    WselState* ws, int blog, int P, const unsigned long long* ngood, unsigned int* err)
{
    const WKey kf(total, n);
    for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x)
        atomicAdd(&ws->hist[kf(absw[i]) >> (24 - blog)], 1u);
    // no start bins yet (the plan marks them)
    for (int b = blockIdx.x * blockDim.x + threadIdx.x; b < (1 << blog); b += gridDim.x * blockDim.x)
        ws->binmap[b] = -1;
    if (last_block(&ws->tickets[0]))
        wsel_plan(ws, blog, n, P, ngood, err);
}

__global__ void __launch_bounds__(256) k_wsel_collect(const double* __restrict__ absw, int64_t n, const double* total,
    WselState* ws, int blog, unsigned long long* mbits, uint32_t* midx)
{
    if (!ws->valid)
        return;
    const WKey kf(total, n);
    for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x) {
        const double a = absw[i];
        const int li = ws->binmap[kf(a) >> (24 - blog)];
        if (li >= 0) {
            const uint32_t pos = ws->list_off[li] + atomicAdd(&ws->cursor[li], 1u);
            mbits[pos] = __double_as_longlong(a);
            midx[pos] = uint32_t(i);
        }
    }
}

// One block per plane p >= 1: the member of the start item's bin whose rank
// under (|w| bits, index) is the wanted one.
__global__ void __launch_bounds__(256) k_wsel_resolve(WselState* ws, const unsigned long long* mbits, const uint32_t* midx)
{
    __shared__ unsigned long long sb[WSEL_CAP];
    __shared__ uint32_t si[WSEL_CAP];
    const int p = blockIdx.x + 1;
    if (!ws->valid)
        return;
    const int li = ws->start_list[p];
    if (li < 0) {
        if (threadIdx.x == 0) {
            ws->start_bits[p] = ~0ull; // after every item: the plane and all later ones are empty
            ws->start_idx[p] = ~0u;
        }
        return;
    }
    const uint32_t off = ws->list_off[li], m = ws->list_cnt[li], want = ws->start_rank[p];
    for (uint32_t e = threadIdx.x; e < m; e += blockDim.x) {
        sb[e] = mbits[off + e];
        si[e] = midx[off + e];
    }
    __syncthreads();
    for (uint32_t e = threadIdx.x; e < m; e += blockDim.x) {
        const unsigned long long b = sb[e];
        const uint32_t ix = si[e];
        uint32_t r = 0;
        for (uint32_t f = 0; f < m; f++)
            r += (sb[f] < b || (sb[f] == b && si[f] < ix)) ? 1u : 0u;
        if (r == want) {
            ws->start_bits[p] = b;
            ws->start_idx[p] = ix;
        }
    }
}

// Plane p's smallest |w| (its start item's; 0 for plane 0) and the fixed-point
// scale of its sums: 2^e with (width * count) * 2^e <= 2^61, width = the
// plane's |w| range (up to the next start item, or wmax).
__device__ __forceinline__ void wsel_range(const WselState* ws, int p, int P, int64_t n, double wmax, double& lo,
    double& scale)
{
    const int64_t cnt = ws->G[p + 1] - ws->G[p];
    lo = p == 0 ? 0.0 : __longlong_as_double((long long)ws->start_bits[p]);
    const double hi = (p + 1 < P && ws->G[p + 1] < n) ? __longlong_as_double((long long)ws->start_bits[p + 1]) : wmax;
    const double span = (hi - lo) * double(cnt);
    if (cnt <= 0 || !(span > 0.0)) {
        scale = 1.0;
        return;
    }
    int ex;
    frexp(span, &ex); // span < 2^ex
    scale = ldexp(1.0, 61 - ex);
}

__global__ void __launch_bounds__(256) k_wsel_classify(const double* __restrict__ absw, int64_t n, int P,
    const double* total, WselState* ws, uint16_t* plane16, unsigned int* err, double* w_avg, int64_t* first)
{
    __shared__ unsigned long long sbits[WSEL_MAXP];
    __shared__ uint32_t sidx[WSEL_MAXP];
    __shared__ double slo[WSEL_MAXP], sscale[WSEL_MAXP];
    // the sums: one copy per warp when the planes fit (less contention on
    // the shared atomics), else one copy for the block
    __shared__ unsigned long long acc[WSEL_MAXP];
    constexpr int kWarpCopyP = WSEL_MAXP / 8;
    const int copies = P <= kWarpCopyP ? 8 : 1;
    if (!ws->valid) {
        // plane 0 for every item: the binning that follows stays in bounds
        // (the host grids again on the sorting path)
        for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x)
            plane16[i] = 0;
        if (blockIdx.x == 0)
            for (int p = threadIdx.x; p < P; p += blockDim.x) {
                w_avg[p] = 0.0;
                first[p] = 0;
            }
        return;
    }
    const double wmax = total[1];
    for (int p = threadIdx.x; p < P; p += blockDim.x) {
        sbits[p] = p == 0 ? 0ull : ws->start_bits[p];
        sidx[p] = p == 0 ? 0u : ws->start_idx[p];
        wsel_range(ws, p, P, n, wmax, slo[p], sscale[p]);
    }
    for (int q = threadIdx.x; q < copies * P; q += blockDim.x)
        acc[q] = 0;
    __syncthreads();
    unsigned long long* myacc = acc + (copies > 1 ? ((threadIdx.x >> 5) & 7) * P : 0);
    bool bad = false;
    for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x) {
        const double a = absw[i];
        if (!(a <= wmax)) { // non-finite |w|
            plane16[i] = 0;
            bad = true;
            continue;
        }
        const unsigned long long b = __double_as_longlong(a);
        const uint32_t ix = uint32_t(i);
        // the last plane whose start item is at or before (b, ix)
        int lo = 0, hi = P - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) / 2;
            if (sbits[mid] < b || (sbits[mid] == b && sidx[mid] <= ix))
                lo = mid;
            else
                hi = mid - 1;
        }
        plane16[i] = uint16_t(lo);
        const double d = a - slo[lo];
        atomicAdd(&myacc[lo], (unsigned long long)rint(d * sscale[lo]));
    }
    if (bad)
        atomicOr(err, 16u);
    __syncthreads();
    for (int p = threadIdx.x; p < P; p += blockDim.x) {
        unsigned long long v = 0;
        for (int c = 0; c < copies; c++)
            v += acc[c * P + p];
        if (v)
            atomicAdd(&ws->sum[p], v);
    }
    // the last block: plane means and starts
    if (last_block(&ws->tickets[1]))
        for (int p = threadIdx.x; p < P; p += blockDim.x) {
            const int64_t cnt = ws->G[p + 1] - ws->G[p];
            w_avg[p] = cnt > 0 ? slo[p] + (double(__ldcg(&ws->sum[p])) / sscale[p]) / double(cnt) : 0.0;
            first[p] = ws->G[p];
        }
}

// The |w| order from a stable sort on the 24-bit keys of k_wkey24 is exact
// except inside runs of equal keys, whose members are in index order.  Each
// run is re-sorted by the full 64-bit key (the bits of |w|), keeping index
// order among equal |w|: the result is the stable order of the 64-bit sort.  Runs longer than kFixRun whose |w| are not all equal set
// bit 4 of *err (the caller then repeats the step with the 64-bit sort).
constexpr int kFixRun = 32;
__global__ void k_fix_runs(const uint32_t* __restrict__ key32, uint32_t* perm, const unsigned long long* __restrict__ key64,
    int64_t n, unsigned int* err)
{
    const int64_t k = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (k + 1 >= n)
        return;
    const uint32_t kk = key32[k];
    if ((k > 0 && key32[k - 1] == kk) || key32[k + 1] != kk)
        return; // not the start of a run of length >= 2
    int64_t e = k + 2;
    while (e < n && e - k <= kFixRun && key32[e] == kk)
        e++;
    const int len = int(e - k);
    if (len == 2) { // the common run: one compare, no per-thread arrays
        const uint32_t p0 = perm[k], p1 = perm[k + 1];
        if (key64[p1] < key64[p0]) {
            perm[k] = p1;
            perm[k + 1] = p0;
        }
        return;
    }
    if (len > kFixRun) {
        const unsigned long long first = key64[perm[k]];
        for (int64_t j = k + 1; j < n && key32[j] == kk; j++)
            if (key64[perm[j]] != first) {
                atomicOr(err, 4u);
                return;
            }
        return; // all |w| equal: index order is already the stable order
    }
    unsigned long long kv[kFixRun];
    uint32_t pv[kFixRun];
    for (int a = 0; a < len; a++) {
        pv[a] = perm[k + a];
        kv[a] = key64[pv[a]];
    }
    // insertion sort by (key64, index): stable, so equal keys keep index order
    for (int a = 1; a < len; a++) {
        const unsigned long long x = kv[a];
        const uint32_t y = pv[a];
        int b = a - 1;
        while (b >= 0 && kv[b] > x) {
            kv[b + 1] = kv[b];
            pv[b + 1] = pv[b];
            b--;
        }
        kv[b + 1] = x;
        pv[b + 1] = y;
    }
    for (int a = 0; a < len; a++)
        perm[k + a] = pv[a];
}

// W-kernel generation for one plane per CTA (FP64), the non-Hankel path of
// WideFieldImaging (aw_projection.cpp:50-111 image-domain kernel with
// combine_2d_kernel_value :455-474, forward c2c FFT :194, truncation
// :197-209, kernel cache :415-448).
//
// The image-domain kernel comb(a, b) is even in both indices (the reference
// writes each value at (+-a, +-b)), non-zero only for |a|, |b| < half, so its
// forward DFT is the separable cosine sum
//   conv(k, l) = sum_{a,b >= 0} m_a m_b Q[a][b] cos(2 pi k a / arr) cos(2 pi l b / arr)
// with m_0 = 1, m_{>0} = 2, and conv(+-k, +-l) = conv(|k|, |l|).  Only the
// entries the cache samples are formed: first the l = 0 row for the
// truncation, then the |offset| block of the truncated support.
// Outputs per plane: support and conv quadrant conv[p][l][k] (stride lh_max),
// from which k_wk_expand forms the cached kernels.
struct WkParams {
    const double* w_avg;
    const double* aa; // image-domain AA kernel over the workarea
    const double* ctab; // cos(2 pi t / arr), t < arr
    int half, arr, os, cs, max_support, lh_max;
    int smem_ctab, smem_Q, smem_T; // k_wkernel_plane: what the launch's dynamic shared memory holds
    double scaled_cell, trunc_perc;
    double2* Qs;   // [P][half][half] from k_wk_quadrant, without smem_Q
    double2* Ts;   // scratch [P][CTAs of a plane][rows of T of a CTA][half], without smem_T
    double2* convd; // [P][lh_max][lh_max] FP64
    int* support;
};

__device__ __forceinline__ double2 wk_value(const WkParams& q, double w, int px, int py)
{
    const int half = q.half;
    const double dx = double(px) * q.scaled_cell, dy = double(py) * q.scaled_cell;
    const double r2 = dx * dx + dy * dy;
    if (r2 >= 1.0)
        return make_double2(q.aa[half + px] * q.aa[half + py], 0.0);
    const double nn = sqrt(1.0 - r2);
    const double ph = (-2.0 * 3.141592653589793238462643383279502884) * w * (nn - 1.0);
    double sn, cn;
    sincos(ph, &sn, &cn);
    const double re = (cn / nn) * q.aa[half + px];
    const double im = (sn / nn) * q.aa[half + px];
    return make_double2(re * q.aa[half + py], im * q.aa[half + py]);
}

// sum_a m_a V[a * stride] cos(2 pi k a / arr), m_0 = 1, m_{>0} = 2
__device__ __forceinline__ double2 cos_sum(const double2* V, int stride, int half, const double* ct, int k, int arr)
{
    double re = 0.0, im = 0.0;
    int at = 0; // k a mod arr
#pragma unroll 4
    for (int a = 0; a < half; a++) {
        const double c = (a == 0 ? 1.0 : 2.0) * ct[at];
        const double2 v = V[size_t(a) * stride];
        re += v.x * c;
        im += v.y * c;
        at += k;
        at = at >= arr ? at - arr : at;
    }
    return make_double2(re, im);
}

// Value (a, b) of the image-domain quadrant, t = a + b half.
__device__ __forceinline__ double2 wk_quadrant(const WkParams& q, double w, int t)
{
    const int a = t % q.half, b = t / q.half;
    if (a == 0 && b == 0)
        return make_double2(q.aa[q.half] * q.aa[q.half], 0.0);
    if (b == 0)
        return wk_value(q, w, a, 0);
    if (a == 0)
        return wk_value(q, w, b, 0); // output(0, i) reuses value(i, 0)
    return wk_value(q, w, a, b);
}

// The quadrants that shared memory does not hold, one for all the CTAs of a
// plane (blockIdx.y): a copy for each would take four times the memory, 8.6 GB
// instead of 2.1 for 32 planes on a workarea of 4096.
__global__ void __launch_bounds__(256) k_wk_quadrant(WkParams q)
{
    const int t = int(blockIdx.x) * 256 + int(threadIdx.x);
    if (t < q.half * q.half)
        q.Qs[size_t(blockIdx.y) * q.half * q.half + t] = wk_quadrant(q, q.w_avg[blockIdx.y], t);
}

// A plane's steps are a chain of short sums, so latency bounds them: the
// cosine table, the image-domain quadrant Q and its row transforms T are kept
// in shared memory where they fit (q.smem_*; the launch gives the room), the
// position in the cosine table is carried instead of reduced modulo arr at
// every term, and the truncation test runs in all threads.  gridDim.y CTAs
// share a plane: each forms Q (in shared memory) and the truncation, then the
// rows l = blockIdx.y, + gridDim.y, ... of T and of the kernel (at support 16
// the kernel's 133^2 sums are most of the work: 193 us with one CTA a plane).
__global__ void __launch_bounds__(1024) k_wkernel_plane(WkParams q)
{
    const int p = blockIdx.x;
    const int half = q.half, arr = q.arr, os = q.os, lh = q.lh_max;
    const double w = q.w_avg[p];
    __shared__ double2 row0[1024];
    __shared__ int s_support;
    extern __shared__ __align__(16) double sct[];
    // 16-byte cells first, then the cosine table
    const int lrows = (lh + int(gridDim.y) - 1) / int(gridDim.y); // rows of T of this CTA, at most
    const size_t cta = size_t(p) * gridDim.y + blockIdx.y;
    double2* sm = reinterpret_cast<double2*>(sct);
    double2* Q = q.Qs + size_t(p) * half * half;
    double2* T = q.Ts + cta * lrows * half;
    if (q.smem_Q) {
        Q = sm;
        sm += size_t(half) * half;
    }
    if (q.smem_T) {
        T = sm;
        sm += size_t(lrows) * half;
    }
    double2* conv = q.convd + size_t(p) * lh * lh;
    const double* ct = q.ctab;
    if (q.smem_ctab) {
        double* sc = reinterpret_cast<double*>(sm);
        for (int t = threadIdx.x; t < arr; t += blockDim.x)
            sc[t] = q.ctab[t];
        ct = sc;
    }
    // 1. image-domain quadrant Q[a][b] (row a, column b)
    if (q.smem_Q)
        for (int t = threadIdx.x; t < half * half; t += blockDim.x)
            Q[t] = wk_quadrant(q, w, t);
    if (threadIdx.x == 0)
        s_support = 0;
    __syncthreads();
    // 2. T[0][a] = sum_b m_b Q[a][b]
    for (int a = threadIdx.x; a < half; a += blockDim.x)
        T[a] = cos_sum(Q + a, half, half, ct, 0, arr);
    __syncthreads();
    // 3. conv(k, 0) at k = i*os for the truncation (k <= arr/2)
    const int kmax0 = min(q.max_support * os, arr >> 1);
    const int nrow = kmax0 / os + 1;
    for (int t = threadIdx.x; t < nrow && t < 1024; t += blockDim.x)
        row0[t] = cos_sum(T, 1, half, ct, t * os, arr);
    __syncthreads();
    if (q.trunc_perc > 0.0) {
        // the last sample above the threshold (0 when none is)
        const double minv = hypot(row0[0].x, row0[0].y) * (q.trunc_perc / 100.0);
        for (int t = 1 + threadIdx.x; t < nrow && t < 1024; t += blockDim.x)
            if (hypot(row0[t].x, row0[t].y) > minv)
                atomicMax(&s_support, t);
    } else if (threadIdx.x == 0) {
        s_support = q.max_support;
    }
    __syncthreads();
    const int S = min(s_support, q.max_support);
    if (threadIdx.x == 0 && blockIdx.y == 0)
        q.support[p] = S;
    const int L = min(S * os + os / 2 + 1, (arr >> 1) + 1);
    // 4. T[l][a] for this CTA's l < L
    const int l0 = int(blockIdx.y), dl = int(gridDim.y);
    const int nl = l0 < L ? (L - l0 + dl - 1) / dl : 0;
    for (int t = threadIdx.x; t < nl * half; t += blockDim.x) {
        const int a = t % half, i = t / half;
        T[size_t(i) * half + a] = cos_sum(Q + a, half, half, ct, l0 + i * dl, arr);
    }
    __syncthreads();
    // 5. conv(k, l) for k < L
    for (int t = threadIdx.x; t < nl * L; t += blockDim.x) {
        const int k = t % L, i = t / L;
        conv[size_t(l0 + i * dl) * lh + k] = cos_sum(T + size_t(i) * half, 1, half, ct, k, arr);
    }
}

// Hankel-transform W-kernels (hankel_opt, aw_projection.cpp:211-287 and
// RadialInterpolate, aw_projection.h:126-214): the radially symmetric W-kernel
// comes from a 1-D transform of the image-domain kernel's radial profile,
// interpolated at the radius of every kernel offset.
struct HankelParams {
    int n;          // radial samples: arr/2 (discrete Hankel transform) or arr (projection slice)
    int proj_slice; // hankel_proj_slice: 1-D DFT of the kernel's projection onto one axis
    int cubic;      // InterpType::CUBIC: natural cubic spline; otherwise linear
    double2* R;     // scratch [P][half]: radial profile or projection
    double2* Y;     // scratch [P][n]: transform at radii 0..n-1 (oversampled uv pixels)
    double2* B;     // scratch [P][n]: spline quadratic coefficients
    double* Cp;     // scratch [P][2][n]: forward-sweep factors of the spline solve
};

// Cubic (natural boundary, tk::spline semantics) or linear interpolation of
// the unit-spaced samples Y at radius r; k = min(floor(r), n - 1), beyond the
// last sample the end segment extrapolates linearly.
__device__ __forceinline__ double2 hankel_interp(const HankelParams& h, const double2* Y, const double2* B, double r)
{
    const int n = h.n;
    const int k = min(int(r), n - 1);
    const double t = r - double(k);
    const double2 y = Y[k];
    if (!h.cubic) {
        const double2 y0 = k < n - 1 ? y : Y[n - 2];
        const double2 y1 = k < n - 1 ? Y[k + 1] : Y[n - 1];
        return make_double2((y1.x - y0.x) * t + y.x, (y1.y - y0.y) * t + y.y);
    }
    auto coef = [&](int i, double2& a, double2& b, double2& c) { // segment i < n - 1
        const double2 b0 = B[i], b1 = B[i + 1], y0 = Y[i], y1 = Y[i + 1];
        a = make_double2(1.0 / 3.0 * (b1.x - b0.x), 1.0 / 3.0 * (b1.y - b0.y));
        b = b0;
        c = make_double2((y1.x - y0.x) - 1.0 / 3.0 * (2.0 * b0.x + b1.x),
                         (y1.y - y0.y) - 1.0 / 3.0 * (2.0 * b0.y + b1.y));
    };
    double2 a, b, c;
    if (k < n - 1) {
        coef(k, a, b, c);
    } else {
        // end segment: a = 0, b = b[n-1] (0 for the natural spline), c = derivative at the last node
        double2 a2, b2, c2;
        coef(n - 2, a2, b2, c2);
        a = make_double2(0.0, 0.0);
        b = B[n - 1];
        c = make_double2(3.0 * a2.x + 2.0 * b2.x + c2.x, 3.0 * a2.y + 2.0 * b2.y + c2.y);
    }
    return make_double2(((a.x * t + b.x) * t + c.x) * t + y.x, ((a.y * t + b.y) * t + c.y) * t + y.y);
}

// One block per W-plane.  Writes the plane's support and its quadrant
// conv[|dy| * lh + |dx|] = f(sqrt(dx^2 + dy^2)), the same outputs as
// k_wkernel_plane.
__global__ void __launch_bounds__(1024) k_hankel_plane(WkParams q, HankelParams h)
{
    const int p = blockIdx.x;
    const int half = q.half, arr = q.arr, os = q.os, lh = q.lh_max, n = h.n;
    const double w = q.w_avg[p];
    double2* R = h.R + size_t(p) * half;
    double2* Y = h.Y + size_t(p) * n;
    double2* B = h.B + size_t(p) * n;
    double2* conv = q.convd + size_t(p) * lh * lh;
    __shared__ int s_support;
    constexpr double kPi = 3.141592653589793238462643383279502884;
    // 1. radial profile (aw_projection.cpp:226-240) or projection (:113-170)
    for (int j = threadIdx.x; j < half; j += blockDim.x) {
        double2 v;
        if (!h.proj_slice) {
            const double dx = double(j) * q.scaled_cell;
            const double r2 = dx * dx;
            if (r2 >= 1.0) {
                v = make_double2(q.aa[half + j], 0.0);
            } else {
                const double nn = sqrt(1.0 - r2);
                double sn, cn;
                sincos((-2.0 * kPi) * w * (nn - 1.0), &sn, &cn);
                v = make_double2((cn / nn) * q.aa[half + j], (sn / nn) * q.aa[half + j]);
            }
        } else if (j == 0) {
            double re = 0.0, im = 0.0;
            for (int i = 1; i < half; i++) {
                const double2 e = wk_value(q, w, i, 0);
                re += e.x;
                im += e.y;
            }
            v = make_double2(re * 2.0 + q.aa[half] * q.aa[half], im * 2.0);
        } else {
            v = wk_value(q, w, j, 0);
            for (int i = 1; i < half; i++) {
                const double2 e = wk_value(q, w, i, j);
                v.x += e.x * 2.0;
                v.y += e.y * 2.0;
            }
        }
        R[j] = v;
    }
    __syncthreads();
    // 2. transform at radii k < n
    const int jmax = min(half, n);
    for (int k = threadIdx.x; k < n; k += blockDim.x) {
        double re = 0.0, im = 0.0;
        if (!h.proj_slice) {
            // DHT column k (aw_projection.cpp:532-596): annulus j spans
            // [rn_{j-1}, rn_j], rn_j = j + 1/2 except rn_{n-1} = n - 1
            const double kk = (kPi / double(n)) * double(k);
            const double kn = (2.0 * kPi) / kk;
            double prev = 0.0;
            for (int j = 0; j < jmax; j++) {
                const double rn = j == n - 1 ? double(n - 1) : double(j) + 0.5;
                const double F = k == 0 ? kPi * rn * rn : kn * rn * besselj1_ref(kk * rn);
                const double d = j == 0 ? F : F - prev;
                prev = F;
                re += d * R[j].x;
                im += d * R[j].y;
            }
        } else {
            // length-arr DFT of the even projection (fft_fftw_dft_c2c_1d)
            re = R[0].x;
            im = R[0].y;
            for (int t = 1; t < half; t++) {
                const double c = 2.0 * q.ctab[(k * t) % arr];
                re += R[t].x * c;
                im += R[t].y * c;
            }
        }
        Y[k] = make_double2(re, im);
    }
    __syncthreads();
    // 3. truncation (aw_projection.h:135-148)
    if (threadIdx.x == 0) {
        int S = q.max_support;
        if (q.trunc_perc > 0.0) {
            const double minv = hypot(Y[0].x, Y[0].y) * (q.trunc_perc / 100.0);
            int t = q.max_support * os;
            while (t > n - 1)
                t -= os;
            while (t > os) {
                if (hypot(Y[t].x, Y[t].y) > minv)
                    break;
                t -= os;
            }
            S = min(int(ceil(double(t) * (1.0 / double(os)))), q.max_support);
        }
        s_support = S;
        q.support[p] = S;
    }
    // 4. natural cubic spline: b_0 = b_{n-1} = 0 and, for 0 < i < n-1,
    //    b_{i-1}/3 + 4 b_i/3 + b_{i+1}/3 = y_{i+1} - 2 y_i + y_{i-1}
    //    (tridiagonal, forward elimination and back substitution; real and
    //    imaginary parts in two threads)
    if (h.cubic && threadIdx.x < 2) {
        const int comp = threadIdx.x;
        const double* y = reinterpret_cast<const double*>(Y) + comp;
        double* b = reinterpret_cast<double*>(B) + comp;
        double* cp = h.Cp + (size_t(p) * 2 + comp) * n;
        b[0] = 0.0;
        b[2 * (n - 1)] = 0.0;
        double cprev = 0.0, dprev = 0.0;
        for (int i = 1; i <= n - 2; i++) {
            const double rhs = (y[2 * (i + 1)] - y[2 * i]) - (y[2 * i] - y[2 * (i - 1)]);
            const double m = 4.0 / 3.0 - (1.0 / 3.0) * cprev;
            cprev = (1.0 / 3.0) / m;
            dprev = (rhs - (1.0 / 3.0) * dprev) / m;
            cp[i] = cprev;
            b[2 * i] = dprev;
        }
        for (int i = n - 3; i >= 1; i--)
            b[2 * i] -= cp[i] * b[2 * (i + 1)];
    }
    __syncthreads();
    // 5. kernel quadrant at the radius of each offset
    const int S = s_support;
    const int L = min(S * os + os / 2 + 1, lh);
    for (int t = threadIdx.x; t < L * L; t += blockDim.x) {
        const int dx = t % L, dy = t / L;
        const double r = dy == 0 ? double(dx) : (dx == 0 ? double(dy) : sqrt(double(dx * dx + dy * dy)));
        conv[size_t(dy) * lh + dx] = hankel_interp(h, Y, B, r);
    }
}

__global__ void k_cos_table(int arr, double* c)
{
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t < arr)
        c[t] = cospi(2.0 * double(t) / double(arr));
}

// Expanded W-kernel tables for the gridder: one block per (plane, oversampled
// offset pair); entry j*K + i (column j, row i) holds the reference's cached
// kernel value conv(|oy|, |ox|) / sum(Re) (aw_projection.cpp:415-448), formed in
// FP64 and rounded once to R.  Plane p's tables start at off[p] = p * stride,
// or (stride 0) right after those of the planes before; *max_support (zeroed
// before) = the largest support.
constexpr int kExpandThreads = 128;
template <typename R>
__global__ void __launch_bounds__(kExpandThreads) k_wk_expand(const double2* convd, const int* support, int P, int cs, int os,
    int lh, uint32_t stride, typename Cplx<R>::T* out, uint32_t* off, unsigned int* max_support)
{
    const int p = blockIdx.x;
    const int pair = blockIdx.y;
    const int cy = pair / cs, cx = pair % cs;
    uint32_t base = uint32_t(p) * stride;
    for (int q = 0; stride == 0 && q < p; q++) {
        const uint32_t Kq = uint32_t(2 * support[q] + 1);
        base += uint32_t(cs) * uint32_t(cs) * Kq * Kq;
    }
    const int S = support[p];
    if (pair == 0 && threadIdx.x == 0) {
        off[p] = base;
        atomicMax(max_support, unsigned(S));
    }
    const int K = 2 * S + 1;
    const double2* conv = convd + size_t(p) * lh * lh;
    auto at = [&](int t) { // |oy|, |ox| of entry t
        const int i = t % K, j = t / K;
        int oy = (i - S) * os + os / 2 - cy;
        int ox = (j - S) * os + os / 2 - cx;
        oy = oy < 0 ? -oy : oy;
        ox = ox < 0 ? -ox : ox;
        return conv[size_t(oy) * lh + ox];
    };
    __shared__ double part[kExpandThreads / 32];
    double ks = 0.0;
    for (int t = threadIdx.x; t < K * K; t += kExpandThreads)
        ks += at(t).x;
    for (int o = 16; o > 0; o >>= 1)
        ks += __shfl_xor_sync(0xffffffffu, ks, o);
    if ((threadIdx.x & 31) == 0)
        part[threadIdx.x >> 5] = ks;
    __syncthreads();
    ks = 0.0;
    for (int w = 0; w < kExpandThreads / 32; w++)
        ks += part[w];
    const double inv = 1 / ks;
    typename Cplx<R>::T* dst = out + base + uint32_t(pair) * uint32_t(K * K);
    for (int t = threadIdx.x; t < K * K; t += kExpandThreads) {
        const double2 v = at(t);
        typename Cplx<R>::T o;
        o.x = R(v.x * inv);
        o.y = R(v.y * inv);
        dst[t] = o;
    }
}

// Copies of a call's results into page-locked host memory through its device
// address: the na words of a, then the 16-byte units of b that hold the
// first a[count_word] records of rec_bytes each (all nb units when
// count_word < 0), at most nb.
__global__ void k_copy_out(const uint32_t* a, uint32_t* ha, int na, const uint4* b, uint4* hb, int nb,
    int count_word, int rec_bytes)
{
    const int t = int(blockIdx.x * blockDim.x + threadIdx.x), stride = int(gridDim.x * blockDim.x);
    for (int i = t; i < na; i += stride)
        ha[i] = a[i];
    int n = nb;
    if (count_word >= 0)
        n = int(min((uint64_t(a[count_word]) * uint64_t(rec_bytes) + 15) / 16, uint64_t(nb)));
    for (int i = t; i < n; i += stride)
        hb[i] = b[i];
}

__global__ void __launch_bounds__(32) k_pack_scalars(PackArgs k) { pack_scalars(k); }

} // namespace stpgpu
