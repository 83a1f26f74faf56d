// The 2-D complex-to-real transform (fft.cpp:45-135) of power-of-two grids,
// with the crop and normalisation (imager.h:97-150) in its last pass.
#pragma once

#include "imager_kernels.cuh"

namespace stpgpu {

// The twiddle factors of a grid of N = 2 M points, each group contiguous in
// the index that a warp's lanes run over (a table of roots read at strides
// costs up to 32 lines a load):
//   [kTwRoots, + N)        exp(2 pi i k / N)
//   [tw_c2r(N, p), ...)    pass p of the c2r: [q][k], k < 16^p
//   [tw_axis(N, L), ...)   second half of an axis transform of L = 32, 64, 128: [q][k], k < 16
constexpr int kC2rMinLog = 7, kC2rMaxLog = 13; // M: grids of 256 to 16384,
constexpr int kC2rMaxLogF = 12;                // in single precision to 8192
__host__ __device__ constexpr int tw_c2r(int N, int pass) { return pass == 1 ? N : (pass == 2 ? N + 256 : N + 256 + 4096); }
__host__ __device__ constexpr int tw_axis(int N, int L)
{
    return N + 256 + 4096 + 8192 + (L == 32 ? 0 : (L == 64 ? 32 : 96));
}
__host__ __device__ constexpr int tw_size(int N) { return tw_axis(N, 128) + 128; }
// radix of pass p >= 1 of the c2r of M points
__host__ __device__ constexpr int c2r_radix(int logm, int pass)
{
    return logm >= 4 * (pass + 1) ? 16 : 1 << (logm - 4 * pass);
}

template <typename T>
__global__ void k_fft_tables(int N, int logm, typename Cplx<T>::T* out)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= tw_size(N))
        return;
    double num = 0.0, den = 1.0;
    auto pass = [&](int e, int ns, int radix) {
        num = double((e / ns) * (e % ns));
        den = double(ns) * radix;
    };
    if (i < N) {
        num = i;
        den = N;
    } else if (i < tw_c2r(N, 2)) {
        pass(i - tw_c2r(N, 1), 16, c2r_radix(logm, 1));
    } else if (i < tw_c2r(N, 3)) {
        pass(i - tw_c2r(N, 2), 256, logm > 8 ? c2r_radix(logm, 2) : 1);
    } else if (i < tw_axis(N, 32)) {
        pass(i - tw_c2r(N, 3), 4096, logm > 12 ? c2r_radix(logm, 3) : 1);
    } else {
        const int L = i < tw_axis(N, 64) ? 32 : (i < tw_axis(N, 128) ? 64 : 128);
        pass(i - tw_axis(N, L), 16, L / 16);
    }
    double s, c;
    sincospi(2.0 * num / den, &s, &c);
    out[i].x = T(c);
    out[i].y = T(s);
}

template <typename C>
__device__ __forceinline__ C c_add(C a, C b)
{
    a.x += b.x;
    a.y += b.y;
    return a;
}
template <typename C>
__device__ __forceinline__ C c_sub(C a, C b)
{
    a.x -= b.x;
    a.y -= b.y;
    return a;
}
template <typename C>
__device__ __forceinline__ C c_mul(C a, C b)
{
    C r;
    r.x = a.x * b.x - a.y * b.y;
    r.y = a.x * b.y + a.y * b.x;
    return r;
}
template <typename C>
__device__ __forceinline__ C c_muli(C a) // i a
{
    C r;
    r.x = -a.y;
    r.y = a.x;
    return r;
}

// Backward (positive exponent) transforms of a few points in registers,
// natural order in and out.
template <typename C>
__device__ __forceinline__ void fft4(C& a0, C& a1, C& a2, C& a3)
{
    const C s0 = c_add(a0, a2), d0 = c_sub(a0, a2), s1 = c_add(a1, a3), d1 = c_muli(c_sub(a1, a3));
    a0 = c_add(s0, s1);
    a1 = c_add(d0, d1);
    a2 = c_sub(s0, s1);
    a3 = c_sub(d0, d1);
}

template <int R, typename C>
__device__ __forceinline__ void fft_points(C* v)
{
    using T = decltype(v[0].x);
    constexpr double r2 = 0.70710678118654752440, c1 = 0.92387953251128675613, s1 = 0.38268343236508977173;
    auto w = [](double x, double y) {
        C r;
        r.x = decltype(r.x)(x);
        r.y = decltype(r.y)(y);
        return r;
    };
    (void)sizeof(T);
    if constexpr (R == 2) {
        const C a = v[0];
        v[0] = c_add(a, v[1]);
        v[1] = c_sub(a, v[1]);
    } else if constexpr (R == 4) {
        fft4(v[0], v[1], v[2], v[3]);
    } else if constexpr (R == 8) {
        fft4(v[0], v[2], v[4], v[6]);
        fft4(v[1], v[3], v[5], v[7]);
        v[3] = c_mul(v[3], w(r2, r2));
        v[5] = c_muli(v[5]);
        v[7] = c_mul(v[7], w(-r2, r2));
        C o[8];
#pragma unroll
        for (int k = 0; k < 4; k++) {
            o[k] = c_add(v[2 * k], v[2 * k + 1]);
            o[k + 4] = c_sub(v[2 * k], v[2 * k + 1]);
        }
#pragma unroll
        for (int k = 0; k < 8; k++)
            v[k] = o[k];
    } else {
        static_assert(R == 16, "radix");
#pragma unroll
        for (int c = 0; c < 4; c++)
            fft4(v[c], v[c + 4], v[c + 8], v[c + 12]);
        // v[c + 4 k1] *= w16^(c k1)
        v[5] = c_mul(v[5], w(c1, s1));
        v[9] = c_mul(v[9], w(r2, r2));
        v[13] = c_mul(v[13], w(s1, c1));
        v[6] = c_mul(v[6], w(r2, r2));
        v[10] = c_muli(v[10]);
        v[14] = c_mul(v[14], w(-r2, r2));
        v[7] = c_mul(v[7], w(s1, c1));
        v[11] = c_mul(v[11], w(-r2, r2));
        v[15] = c_mul(v[15], w(-c1, -s1));
        C o[16];
#pragma unroll
        for (int k = 0; k < 4; k++) {
            fft4(v[4 * k], v[4 * k + 1], v[4 * k + 2], v[4 * k + 3]);
#pragma unroll
            for (int q = 0; q < 4; q++)
                o[k + 4 * q] = v[4 * k + q];
        }
#pragma unroll
        for (int k = 0; k < 16; k++)
            v[k] = o[k];
    }
}

// ---------------------------------------------------------------- columns axis

// The backward transform along the grid's columns (length N = N1 N2, element
// stride ld) in two passes over the grid, in place: with n = N2 n1 + n2 and k
// = k1 + N1 k2, pass A transforms over n1 for every n2, multiplies by
// exp(2 pi i n2 k1 / N) and leaves k1 in the place of n1; pass B transforms
// over n2 for every k1 and leaves k2 in the place of n2.  Value k is then in
// column axis_place(k).  A CTA takes L columns x 32 rows: lanes are rows, so
// every access is a run of 32 cells; a thread holds 16 of the L points, and
// the rest of the transform exchanges through shared memory.  Both passes
// read and write the grid once: the bound is HBM.
__host__ __device__ constexpr int axis_n1(int N) { return N >= 8192 ? 128 : (N >= 2048 ? 64 : (N >= 512 ? 32 : 16)); }
__host__ __device__ __forceinline__ int axis_place(int k, int N)
{
    const int n1 = axis_n1(N), n2 = N / n1;
    return n2 * (k & (n1 - 1)) + k / n1;
}
__host__ __device__ constexpr int axis_groups(int L) { return L >= 64 ? 1 : 128 / (L * 2); } // transforms per CTA: 128 threads or more
__host__ __device__ constexpr int axis_threads(int L) { return 32 * (L / 16) * axis_groups(L); }

template <typename T, int L, bool FIRST>
__global__ void __launch_bounds__(axis_threads(L), sizeof(T) == 8 ? 512 / axis_threads(L) : 768 / axis_threads(L))
    k_fft_axis(typename Cplx<T>::T* __restrict__ g, int ld, int rows, int N, const typename Cplx<T>::T* __restrict__ tw)
{
    using C = typename Cplx<T>::T;
    constexpr int TL = L / 16, G = axis_groups(L);
    extern __shared__ __align__(16) unsigned char smem_fft[];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int t = w % TL, slot = w / TL;
    C* sm = reinterpret_cast<C*>(smem_fft) + slot * (L * 32);
    const int other = N / L; // the other factor
    const int grp = int(blockIdx.y) * G + slot;
    const int row = int(blockIdx.x) * 32 + lane;
    const bool live = row < rows;
    // column of point m: FIRST other * m + grp, else L * grp + m
    const size_t step = FIRST ? size_t(other) * size_t(ld) : size_t(ld);
    C* base = g + (FIRST ? size_t(grp) : size_t(L) * size_t(grp)) * size_t(ld) + size_t(live ? row : 0);
    // (lanes beyond the last row read nothing: other blocks write the cells of every row there is)
    C v[16] = {};
    if (live) {
#pragma unroll
        for (int q = 0; q < 16; q++)
            v[q] = base[size_t(t + q * TL) * step];
    }
    fft_points<16>(v);
    if constexpr (TL > 1) {
#pragma unroll
        for (int q = 0; q < 16; q++)
            sm[(t * 16 + q) * 32 + lane] = v[q];
        __syncthreads();
        const C* ta = tw + tw_axis(N, L);
#pragma unroll
        for (int b = 0; b < 16 / TL; b++) {
            const int k = t + b * TL; // < 16
#pragma unroll
            for (int q = 0; q < TL; q++) {
                v[b * TL + q] = sm[(k + q * 16) * 32 + lane];
                if (q > 0)
                    v[b * TL + q] = c_mul(v[b * TL + q], __ldg(ta + q * 16 + k));
            }
            fft_points<TL>(v + b * TL);
        }
    }
    if (!live)
        return;
#pragma unroll
    for (int b = 0; b < 16 / TL; b++)
#pragma unroll
        for (int q = 0; q < TL; q++) {
            const int m = TL > 1 ? t + b * TL + q * 16 : b;
            C x = v[b * TL + q];
            if (FIRST)
                x = c_mul(x, __ldg(tw + grp * m));
            base[size_t(m) * step] = x;
        }
}

// ---------------------------------------------------------------- c2r

// cos and sin of 2 pi q / 32, q < 16
__host__ __device__ constexpr double cos_32(int q)
{
    constexpr double c[9] = { 1.0, 0.98078528040323044913, 0.92387953251128675613, 0.83146961230254523708,
        0.70710678118654752440, 0.55557023301960222474, 0.38268343236508977173, 0.19509032201612826785, 0.0 };
    return q <= 8 ? c[q] : -c[16 - q];
}
__host__ __device__ constexpr double sin_32(int q) { return q <= 8 ? cos_32(8 - q) : cos_32(q - 8); }

// One output column: the complex-to-real transform of N points from its
// N/2 + 1 spectrum values, scaled and cropped on the way out.  The even and
// odd samples are packed as one complex sequence of M = N/2 points, which a
// thread group of M/16 transforms with 16 points a thread: radix-16 passes
// (and one smaller) that exchange through shared memory, so a 4096-point
// column crosses it twice.  The spectrum is read once and the image written
// once: the bound is HBM (double columns of 8192: about even with the FP64
// pipe), with 24 warps an SM in single and 16 in double precision to hide the
// exchanges' latency.  cuFFT's own c2r writes the padded image in one or two
// passes and the normalisation reads and writes it again: 52 us on 4096^2
// single, 116 double, 471 on 8192^2 double, here 42, 70 and 246 (with the
// passes along the columns 76, 153 and 600 against 103, 201 and 808).
__host__ __device__ constexpr int c2r_rows(int logm) { return logm >= 12 ? 1 : (4096 >> logm); } // columns per block
__host__ __device__ constexpr int c2r_threads(int logm) { return ((1 << logm) / 16) * c2r_rows(logm); }
__host__ __device__ constexpr size_t c2r_smem(int logm, size_t cell)
{
    return size_t(c2r_rows(logm)) * ((size_t(1) << logm) + (size_t(1) << logm) / 16) * cell;
}

template <int R, int LOGM, int NS, typename C>
__device__ __forceinline__ void c2r_pass(C* v, const C* sm, const C* __restrict__ tw, int t)
{
    constexpr int M = 1 << LOGM, T16 = M / 16;
#pragma unroll
    for (int b = 0; b < 16 / R; b++) {
        const int tb = t + b * T16;
        const int k = tb & (NS - 1);
#pragma unroll
        for (int q = 0; q < R; q++) {
            const int i = tb + q * (M / R);
            v[b * R + q] = sm[i + (i >> 4)];
            if (q > 0)
                v[b * R + q] = c_mul(v[b * R + q], __ldg(tw + q * NS + k));
        }
        fft_points<R>(v + b * R);
    }
}

template <int LOGM, int NS, typename C>
__device__ __forceinline__ void c2r_store(const C* v, C* sm, int t)
{
    const int k = t & (NS - 1);
    const int d = (t - k) * 16 + k;
#pragma unroll
    for (int q = 0; q < 16; q++) {
        const int i = d + q * NS;
        sm[i + (i >> 4)] = v[q];
    }
}

template <typename T, typename RO, int LOGM>
__global__ void __launch_bounds__(c2r_threads(LOGM), sizeof(T) == 8 ? (LOGM == 13 ? 1 : 2) : 3)
    k_c2r_normalise(const typename Cplx<T>::T* __restrict__ F, int ld, const typename Cplx<T>::T* __restrict__ tw,
        int image_size, const double* total, const double* __restrict__ ginv, int corr, RO* __restrict__ out, PackArgs pk)
{
    using C = typename Cplx<T>::T;
    constexpr int M = 1 << LOGM, N = 2 * M, T16 = M / 16;
    extern __shared__ __align__(16) unsigned char smem_fft[];
    if (pk.out && blockIdx.x == 0 && threadIdx.x < 32)
        pack_scalars(pk);
    const int t = threadIdx.x % T16, slot = threadIdx.x / T16;
    C* sm = reinterpret_cast<C*>(smem_fft) + slot * (M + M / 16);
    const int hp = N / 2, hs = image_size / 2;
    const int jo = int(blockIdx.x) * c2r_rows(LOGM) + slot; // output column
    const bool live = jo < image_size;
    const int j = !live ? 0 : (jo < hs ? jo : N + jo - image_size);
    const C* f = F + size_t(axis_place(j, N)) * size_t(ld);
    C v[16];
#pragma unroll
    for (int q = 0; q < 16; q++)
        v[q] = __ldg(f + t + q * T16);
    C last = v[0];
    if (t == 0)
        last = __ldg(f + M);
    // the partners F[M - k] through shared memory: read from global memory
    // they miss L1 half the time and double the traffic from L2
#pragma unroll
    for (int q = 0; q < 16; q++) {
        const int k = t + q * T16;
        sm[k + (k >> 4)] = v[q];
    }
    __syncthreads();
    // Z[k] = E[k] + i O[k], E = F[k] + conj F[M - k], O = (F[k] - conj F[M - k]) e^(2 pi i k / N)
    const C wt = __ldg(tw + t);
#pragma unroll
    for (int q = 0; q < 16; q++) {
        const int k = t + q * T16, kp = q == 0 && t == 0 ? 0 : M - k;
        C a = v[q], b = sm[kp + (kp >> 4)], w;
        if (q == 0 && t == 0) {
            b = last;
            a.y = b.y = T(0); // real by symmetry: their imaginary parts do not enter
        }
        if (sizeof(T) == 8) { // e^(2 pi i t / N) e^(2 pi i q / 32): the table does not stay in L1
            C cq;
            cq.x = T(cos_32(q));
            cq.y = T(sin_32(q));
            w = c_mul(wt, cq);
        } else {
            w = __ldg(tw + k);
        }
        C e, d;
        e.x = a.x + b.x;
        e.y = a.y - b.y;
        d.x = a.x - b.x;
        d.y = a.y + b.y;
        const C o = c_mul(d, w);
        v[q].x = e.x - o.y;
        v[q].y = e.y + o.x;
    }
    __syncthreads();
    fft_points<16>(v);
    c2r_store<LOGM, 1>(v, sm, t);
    __syncthreads();
    constexpr int kPasses = (LOGM + 3) / 4; // after the first: kPasses - 1
    if constexpr (kPasses > 2) {
        c2r_pass<16, LOGM, 16>(v, sm, tw + tw_c2r(N, 1), t);
        __syncthreads();
        c2r_store<LOGM, 16>(v, sm, t);
        __syncthreads();
    }
    if constexpr (kPasses > 3) {
        c2r_pass<16, LOGM, 256>(v, sm, tw + tw_c2r(N, 2), t);
        __syncthreads();
        c2r_store<LOGM, 256>(v, sm, t);
        __syncthreads();
    }
    constexpr int RL = c2r_radix(LOGM, kPasses - 1), NL = 1 << (4 * (kPasses - 1));
    static_assert(RL * NL == M, "passes");
    c2r_pass<RL, LOGM, NL>(v, sm, tw + tw_c2r(N, kPasses - 1), t);
    if (!live)
        return;
    const double tot = total[0];
    const double nf = tot > 0.0 ? 1.0 / tot : 0.0;
    const double fj = corr ? nf * ginv[(j + hp) & (N - 1)] : nf;
    RO* dst = out + size_t(jo) * size_t(image_size);
    auto scaled = [&](C z, int i, double& x, double& y) { // samples i and i + 1
        x = double(z.x) * fj;
        y = double(z.y) * fj;
        if (corr) {
            const double2 g = __ldg(reinterpret_cast<const double2*>(ginv + ((i + hp) & (N - 1))));
            x *= g.x;
            y *= g.y;
        }
    };
    auto pair = [](double x, double y) {
        typename Cplx<RO>::T o;
        o.x = RO(x);
        o.y = RO(y);
        return o;
    };
    if (image_size == N) {
#pragma unroll
        for (int b = 0; b < 16 / RL; b++)
#pragma unroll
            for (int q = 0; q < RL; q++) {
                const int m = t + b * T16 + q * (M / RL);
                double x, y;
                scaled(v[b * RL + q], 2 * m, x, y);
                reinterpret_cast<typename Cplx<RO>::T*>(dst)[m] = pair(x, y);
            }
        return;
    }
#pragma unroll
    for (int b = 0; b < 16 / RL; b++)
#pragma unroll
        for (int q = 0; q < RL; q++) {
            const int i = 2 * (t + b * T16 + q * (M / RL));
            const bool in0 = i < hs || i >= N - hs, in1 = i + 1 < hs || i + 1 >= N - hs;
            if (!in0 && !in1)
                continue;
            double x, y;
            scaled(v[b * RL + q], i, x, y);
            if (in0 && in1) // i and the crop's offset are even: aligned
                *reinterpret_cast<typename Cplx<RO>::T*>(dst + (i < hs ? i : i + image_size - N)) = pair(x, y);
            else if (in0)
                dst[i < hs ? i : i + image_size - N] = RO(x);
            else
                dst[i + 1 < hs ? i + 1 : i + 1 + image_size - N] = RO(y);
        }
}

} // namespace stpgpu
