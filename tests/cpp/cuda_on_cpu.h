// Runs a kernel's source on the CPU, a thread per CUDA thread and the blocks
// one after the other, for checks of a kernel's memory accesses.  The test
// that includes it replaces `extern __shared__` by `extern` and `__shared__`
// by `static` in the kernel's text.
#pragma once

#include <barrier>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <memory>
#include <mutex>
#include <thread>
#include <utility>
#include <vector>

#define __global__
#define __device__
#define __host__
#define __forceinline__ inline
#define __launch_bounds__(...)
#define __align__(n) __attribute__((aligned(n)))

struct float2 {
    float x, y;
};
struct double2 {
    double x, y;
};
struct Dim3 {
    unsigned x = 1, y = 1, z = 1;
};

inline thread_local Dim3 threadIdx;
inline Dim3 blockIdx, blockDim, gridDim;
inline std::unique_ptr<std::barrier<>> block_barrier;
inline std::vector<std::unique_ptr<std::barrier<>>> warp_barriers;

inline void __syncthreads() { block_barrier->arrive_and_wait(); }
inline void __syncwarp() { warp_barriers[threadIdx.x / 32]->arrive_and_wait(); }
// every lane of a warp takes part
inline std::vector<std::vector<uint64_t>> warp_slots;
template <typename T>
T __shfl_sync(unsigned, T v, int from)
{
    auto& slots = warp_slots[threadIdx.x / 32];
    __builtin_memcpy(&slots[threadIdx.x % 32], &v, sizeof(T));
    __syncwarp();
    T r;
    __builtin_memcpy(&r, &slots[from], sizeof(T));
    __syncwarp();
    return r;
}
inline unsigned __ballot_sync(unsigned, bool v)
{
    auto& slots = warp_slots[threadIdx.x / 32];
    slots[threadIdx.x % 32] = v;
    __syncwarp();
    unsigned r = 0;
    for (int i = 0; i < 32; i++)
        r |= unsigned(slots[i] != 0) << i;
    __syncwarp();
    return r;
}
inline int __ffs(int v) { return __builtin_ffs(v); }
template <typename T>
inline T __ldg(const T* p)
{
    return *p;
}
inline double __dadd_rn(double a, double b) { return a + b; }
inline double __dmul_rn(double a, double b) { return a * b; }
inline uint32_t min(uint32_t a, uint32_t b) { return a < b ? a : b; }
inline void sincospi(double x, double* s, double* c)
{
    *s = std::sin(M_PI * x);
    *c = std::cos(M_PI * x);
}

template <typename F>
void launch(Dim3 grid, unsigned threads, F kernel)
{
    gridDim = grid;
    blockDim = Dim3 { threads, 1, 1 };
    for (unsigned by = 0; by < grid.y; by++)
        for (unsigned bx = 0; bx < grid.x; bx++) {
            blockIdx = Dim3 { bx, by, 0 };
            block_barrier = std::make_unique<std::barrier<>>(threads);
            warp_barriers.clear();
            warp_slots.assign((threads + 31) / 32, std::vector<uint64_t>(32));
            for (unsigned w = 0; w < threads; w += 32)
                warp_barriers.push_back(std::make_unique<std::barrier<>>(std::min(32u, threads - w)));
            std::vector<std::thread> pool;
            for (unsigned t = 0; t < threads; t++)
                pool.emplace_back([&kernel, t] {
                    threadIdx = Dim3 { t, 0, 0 };
                    kernel();
                    // threads that have returned are not waited for
                    block_barrier->arrive_and_drop();
                    warp_barriers[t / 32]->arrive_and_drop();
                });
            for (auto& t : pool)
                t.join();
        }
}
