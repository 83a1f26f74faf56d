// Host orchestration and the extern "C" layer (include/stpgpu.h).
//
// One stpgpu_context = one device + one stream + cached scratch buffers and
// cuFFT plans.  An entry point enqueues its whole pipeline on the context
// stream and synchronises once at the end to read back the few scalars the
// caller needs.
#include <cub/cub.cuh>
#include <cufft.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <initializer_list>
#include <iterator>
#include <utility>
#include <cstdlib>
#include <cstring>
#include <functional>
#include <map>
#include <set>
#include <unordered_map>
#include <chrono>
#include <thread>
#include <memory>
#include <deque>
#include <condition_variable>
#include <mutex>
#include <string>
#include <tuple>
#include <type_traits>
#include <vector>

#include "common.cuh"
#include "imager_kernels.cuh"
#include "gridder_kernels.cuh"
#include "fft_kernels.cuh"
#include "sourcefind_kernels.cuh"
#include "visibility_kernels.cuh"
#include "aproj_kernels.cuh"

using namespace stpgpu;

namespace {
// Zeroes ranges of 32-bit words (at most four) with one kernel launch.
void zero_words(cudaStream_t st, std::initializer_list<std::pair<void*, int64_t>> ranges)
{
    ZeroRanges z {};
    int64_t most = 0;
    int r = 0;
    for (const auto& q : ranges) {
        z.p[r] = static_cast<uint32_t*>(q.first);
        z.n[r] = q.second;
        most = std::max(most, q.second);
        r++;
    }
    const unsigned blocks = unsigned(std::min<int64_t>(std::max<int64_t>((most + 255) / 256, 1), 148 * 4));
    k_zero_ranges<<<blocks, 256, 0, st>>>(z);
    STPGPU_CHECK_LAUNCH();
}

// A captured graph with its zero-filling memset nodes (the library's own
// scratch clears, e.g. CUB's) replaced by k_zero_ranges kernel nodes: a
// replayed graph spends 2-5 us of idle time at a memset node, about 0.1 us
// at a kernel node.  Works on a clone; returns the clone, or the original
// graph when a node cannot be rewritten (nothing is changed then);
// *added = the kernel nodes added.
cudaGraph_t memsets_to_kernels(cudaGraph_t graph, int* added)
{
    *added = 0;
    size_t count = 0;
    if (cudaGraphGetNodes(graph, nullptr, &count) != cudaSuccess || count == 0)
        return graph;
    cudaGraph_t clone = nullptr;
    if (cudaGraphClone(&clone, graph) != cudaSuccess)
        return graph;
    auto give_up = [&] {
        cudaGraphDestroy(clone);
        (void)cudaGetLastError();
        *added = 0;
        return graph;
    };
    std::vector<cudaGraphNode_t> nodes(count);
    if (cudaGraphGetNodes(clone, nodes.data(), &count) != cudaSuccess)
        return give_up();
    for (cudaGraphNode_t nd : nodes) {
        cudaGraphNodeType type;
        if (cudaGraphNodeGetType(nd, &type) != cudaSuccess)
            return give_up();
        if (type != cudaGraphNodeTypeMemset)
            continue;
        cudaMemsetParams mp {};
        if (cudaGraphMemsetNodeGetParams(nd, &mp) != cudaSuccess)
            return give_up();
        const size_t bytes = size_t(mp.width) * mp.elementSize;
        if (mp.value != 0 || mp.height != 1 || bytes % 4 != 0 || (reinterpret_cast<uintptr_t>(mp.dst) & 3) != 0)
            continue;
        size_t nin = 0, nout = 0;
        if (cudaGraphNodeGetDependencies(nd, nullptr, &nin) != cudaSuccess
            || cudaGraphNodeGetDependentNodes(nd, nullptr, &nout) != cudaSuccess)
            return give_up();
        std::vector<cudaGraphNode_t> in(nin), out(nout);
        if ((nin && cudaGraphNodeGetDependencies(nd, in.data(), &nin) != cudaSuccess)
            || (nout && cudaGraphNodeGetDependentNodes(nd, out.data(), &nout) != cudaSuccess))
            return give_up();
        ZeroRanges z {};
        z.p[0] = static_cast<uint32_t*>(mp.dst);
        z.n[0] = int64_t(bytes / 4);
        void* args[] = { &z };
        cudaKernelNodeParams kp {};
        kp.func = reinterpret_cast<void*>(k_zero_ranges);
        kp.gridDim = dim3(unsigned(std::min<int64_t>(std::max<int64_t>((z.n[0] + 255) / 256, 1), 148 * 4)));
        kp.blockDim = dim3(256);
        kp.sharedMemBytes = 0;
        kp.kernelParams = args;
        cudaGraphNode_t kn = nullptr;
        if (cudaGraphAddKernelNode(&kn, clone, nin ? in.data() : nullptr, nin, &kp) != cudaSuccess)
            return give_up();
        for (cudaGraphNode_t o : out)
            if (cudaGraphAddDependencies(clone, &kn, &o, 1) != cudaSuccess)
                return give_up();
        if (cudaGraphDestroyNode(nd) != cudaSuccess)
            return give_up();
        ++*added;
    }
    cudaGraphDestroy(graph);
    return clone;
}
} // namespace

namespace {
struct DevBuf {
    void* p = nullptr;
    size_t cap = 0;
};

// Words zeroed at the start of a call (GridOut::d_err points at them).
enum CallFlags { CF_ERR = 0, CF_MAX_SUPPORT, CF_RANK_OVERFLOW, CF_ENTRIES, CF_TICKET, CF_WORDS };

// Device outputs of one gridding pass (context buffers).
struct GridOut {
    void* grid = nullptr;
    void* beam = nullptr;
    int image_rows = 0;
    int ld = 0; // cells from one grid column to the next
    double* d_total = nullptr;             // [0] sample_grid_total
    unsigned long long* d_ngood = nullptr; // [0] good visibilities
    uint32_t* d_nitems = nullptr;          // binned entries
    unsigned int* d_err = nullptr;         // error flags, then the other words of CallFlags
    int* d_plane_support = nullptr;
    int nplanes = 0;
};

} // namespace

struct stpgpu_context {
    int device = 0;
    cudaStream_t stream = nullptr;
    cudaEvent_t ev0 = nullptr, ev1 = nullptr;
    bool timing = false;
    cudaEvent_t pev[5] = { nullptr, nullptr, nullptr, nullptr, nullptr };
    std::string err;

    void mark(int k)
    {
        if (timing && pev[k])
            STPGPU_CUDA_TRY(cudaEventRecord(pev[k], stream));
    }
    std::map<std::string, DevBuf> bufs;
    std::map<std::tuple<int, int, cudaStream_t>, cufftHandle> plans; // (N, cufftType, stream)
    std::map<std::tuple<int, int, int, cudaStream_t>, cufftHandle> plans_many; // (N, type, batch, stream)
    // Prefix of buffer and memo names: the batch path gives every snapshot
    // slot its own buffers ("b<i>/"); single calls use "".
    std::string ns;

    // batch path: worker streams, fork/join events, the captured graph of
    // the last batch signature and a pinned staging area (scalar read-back)
    std::vector<cudaStream_t> wstreams;
    std::vector<cudaEvent_t> wevents;
    cudaEvent_t fork_ev = nullptr;
    std::string batch_sig;
    int batch_calls = 0;
    cudaGraph_t batch_graph = nullptr;
    cudaGraphExec_t batch_exec = nullptr;
    void* batch_host = nullptr;
    size_t batch_host_cap = 0;

    // single-call path: graph of the last device-pointer call (see run_imager)
    std::string single_sig;
    cudaGraph_t single_graph = nullptr;
    cudaGraphExec_t single_exec = nullptr;
    GridOut single_g {};
    uint32_t sf_label_cap = 0; // source finder: label-analysis capacities that sufficed so far
    uint32_t sf_fg_cap = 0;
    int single_launches = 0; // our kernels in single_graph (counted at capture)
    int batch_launches = 0;  // our kernels in batch_graph
    // source finder: graph of the first attempt of the last call (see
    // run_source_find); sf_graph_off after a capture that failed
    std::string sf_sig;
    cudaGraph_t sf_graph = nullptr;
    cudaGraphExec_t sf_exec = nullptr;
    int sf_launches = 0;
    bool sf_graph_off = false;
    // size classes whose last single call could not take the W-planes
    // without the |w| sort (their calls sort)
    std::set<std::string> wsel_off;
    // bumped whenever a device buffer or the page-locked stage is
    // reallocated: a captured graph whose signature holds an older value
    // may point at freed memory
    uint64_t buf_gen = 0;

    void drop_sf_graph()
    {
        if (sf_exec)
            cudaGraphExecDestroy(sf_exec);
        if (sf_graph)
            cudaGraphDestroy(sf_graph);
        sf_exec = nullptr;
        sf_graph = nullptr;
        sf_sig.clear();
    }

    void drop_single()
    {
        if (single_exec)
            cudaGraphExecDestroy(single_exec);
        if (single_graph)
            cudaGraphDestroy(single_graph);
        single_exec = nullptr;
        single_graph = nullptr;
        single_sig.clear();
    }

    void drop_graph()
    {
        if (batch_exec)
            cudaGraphExecDestroy(batch_exec);
        if (batch_graph)
            cudaGraphDestroy(batch_graph);
        batch_exec = nullptr;
        batch_graph = nullptr;
    }
    void* pinned = nullptr;
    void* pinned_dev = nullptr; // the device's address of the staging area (mapped)
    size_t pinned_cap = 0;
    std::map<std::string, std::string> memo_keys; // buffer name -> key of its current contents

    // True when buffer `name` already holds the data described by `key`
    // (static tables: gcf, kernel tables, cos tables); records `key`.
    bool memo(const std::string& name, const std::string& key)
    {
        auto it = memo_keys.find(ns + name);
        if (it != memo_keys.end() && it->second == key)
            return true;
        memo_keys[ns + name] = key;
        return false;
    }

    // STPGPU_LOG_ALLOC=1: one line per allocation or plan creation with its
    // host time (allocations after warm-up are what stall a serving loop)
    static void log_alloc(const char* what, const std::string& name, size_t bytes,
        std::chrono::steady_clock::time_point t0)
    {
        static const bool on = std::getenv("STPGPU_LOG_ALLOC") != nullptr;
        if (!on)
            return;
        const double ms = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
        std::fprintf(stderr, "stpgpu alloc: %s %s %zu bytes %.3f ms\n", what, name.c_str(), bytes, ms);
    }

    // Named scratch buffer, grown on demand (steady state allocates nothing).
    template <typename T>
    T* buf(const std::string& name, size_t count)
    {
        const size_t bytes = std::max<size_t>(count * sizeof(T), 256);
        DevBuf& b = bufs[ns + name];
        if (b.cap < bytes) {
            if (b.p) {
                STPGPU_CUDA_TRY(cudaStreamSynchronize(stream));
                STPGPU_CUDA_TRY(cudaFree(b.p));
                b.p = nullptr;
                b.cap = 0;
            }
            const size_t want = bytes + bytes / 8;
            const auto t0 = std::chrono::steady_clock::now();
            buf_gen++;
            STPGPU_CUDA_TRY(cudaMalloc(&b.p, want));
            log_alloc("device buffer", ns + name, want, t0);
            b.cap = want;
            memo_keys.erase(ns + name);
        }
        return reinterpret_cast<T*>(b.p);
    }

    template <typename T>
    T* host_stage(size_t count)
    {
        const size_t bytes = std::max<size_t>(count * sizeof(T), 256);
        if (pinned_cap < bytes) {
            if (pinned) {
                STPGPU_CUDA_TRY(cudaStreamSynchronize(stream));
                cudaFreeHost(pinned);
            }
            pinned = nullptr;
            pinned_dev = nullptr;
            pinned_cap = 0;
            const auto t0 = std::chrono::steady_clock::now();
            buf_gen++;
            STPGPU_CUDA_TRY(cudaHostAlloc(&pinned, bytes, cudaHostAllocMapped));
            STPGPU_CUDA_TRY(cudaHostGetDevicePointer(&pinned_dev, pinned, 0));
            log_alloc("page-locked stage", ns, bytes, t0);
            pinned_cap = bytes;
        }
        return reinterpret_cast<T*>(pinned);
    }

    // The device's address of a location in the staging area: kernels write
    // a call's results there directly (a kernel node in place of a copy node
    // in the captured graphs).
    template <typename T>
    T* host_stage_dev(T* h) const
    {
        return reinterpret_cast<T*>(static_cast<unsigned char*>(pinned_dev)
            + (reinterpret_cast<unsigned char*>(h) - static_cast<unsigned char*>(pinned)));
    }

    // One plan per (size, type, stream): a plan's work area must not be
    // shared by transforms running concurrently on different streams.
    cufftHandle plan(int N, cufftType type)
    {
        const auto key = std::make_tuple(N, int(type), stream);
        auto it = plans.find(key);
        if (it != plans.end())
            return it->second;
        cufftHandle h;
        const auto t0 = std::chrono::steady_clock::now();
        cufftResult r = cufftPlan2d(&h, N, N, type);
        log_alloc("cuFFT plan", ns + "N" + std::to_string(N), 0, t0);
        if (r != CUFFT_SUCCESS)
            fail(STPGPU_ERR_CUFFT, "cufftPlan2d failed (" + std::to_string(int(r)) + ") for N=" + std::to_string(N));
        r = cufftSetStream(h, stream);
        if (r != CUFFT_SUCCESS)
            fail(STPGPU_ERR_CUFFT, "cufftSetStream failed");
        plans[key] = h;
        return h;
    }

    // Batched N x N transforms (A-projection kernels), cached like plan().
    cufftHandle plan_many(int N, cufftType type, int batch)
    {
        const auto key = std::make_tuple(N, int(type), batch, stream);
        auto it = plans_many.find(key);
        if (it != plans_many.end())
            return it->second;
        cufftHandle h;
        int dims[2] = { N, N };
        const auto t0 = std::chrono::steady_clock::now();
        cufftResult r = cufftPlanMany(&h, 2, dims, nullptr, 1, N * N, nullptr, 1, N * N, type, batch);
        log_alloc("cuFFT plan", ns + "N" + std::to_string(N) + "x" + std::to_string(batch), 0, t0);
        if (r != CUFFT_SUCCESS)
            fail(STPGPU_ERR_CUFFT, "cufftPlanMany failed (" + std::to_string(int(r)) + ") for N=" + std::to_string(N));
        r = cufftSetStream(h, stream);
        if (r != CUFFT_SUCCESS)
            fail(STPGPU_ERR_CUFFT, "cufftSetStream failed");
        plans_many[key] = h;
        return h;
    }

    void release()
    {
        if (stream)
            cudaStreamSynchronize(stream);
        for (auto w : wstreams)
            cudaStreamSynchronize(w);
        drop_graph();
        drop_single();
        drop_sf_graph();
        batch_sig.clear();
        batch_calls = 0;
        for (auto& kv : plans)
            cufftDestroy(kv.second);
        plans.clear();
        for (auto& kv : plans_many)
            cufftDestroy(kv.second);
        plans_many.clear();
        for (auto& kv : bufs)
            if (kv.second.p)
                cudaFree(kv.second.p);
        bufs.clear();
        memo_keys.clear();
    }
};

namespace {

std::string fkey(double v)
{
    char b[64];
    std::snprintf(b, sizeof(b), "%a", v);
    return b;
}

constexpr size_t pad256(size_t b) { return (b + 255) / 256 * 256; }
constexpr size_t pad16(size_t b) { return (b + 15) / 16 * 16; }

inline unsigned grid1d(int64_t n, int threads) { return unsigned(std::max<int64_t>(1, ceil_div(n, threads))); }

stpgpu_status guard(stpgpu_context* ctx, const std::function<void()>& f)
{
    if (!ctx)
        return STPGPU_ERR_INVALID_ARG;
    try {
        STPGPU_CUDA_TRY(cudaSetDevice(ctx->device));
        f();
        ctx->err.clear();
        return STPGPU_OK;
    } catch (const Error& e) {
        ctx->err = e.msg;
        if (ctx->stream)
            cudaStreamSynchronize(ctx->stream);
        return e.status;
    } catch (const std::exception& e) {
        ctx->err = e.what();
        return STPGPU_ERR_CUDA;
    }
}

double arc_sec_to_rad(double v) { return (v / 3600.0) * (M_PI / 180.0); } // gridder.h:20

// ------------------------------------------------------------------ imager

struct ImagerSetup {
    int kf = kPSWF;
    double trunc = 0.0; // functor argument
    int support = 0;    // AA kernel support
    int N = 0;          // padded (grid) size
    int kernel_exact = 0;
    int os = 1;
    int shift_uv = 1, halfplane = 1, beam = 0;
    int analytic = 0;
    double cell_size = 0.0;
    int nplanes = 0, max_support = 0, undersampling = 1, wmedian = 0;
    double trunc_perc = 0.0;
    int full_wsort = 0; // |w| order from the 64-bit sort (fallback of the 32-bit sort + run fix-up)
    int wsel = 0;       // W-planes without the |w| sort (k_wsel_*; single calls, falls back through error bit 16)
    int hankel = 0, proj_slice = 0, cubic = 0; // Hankel-transform W-kernels (hankel_opt)
    // A-projection: time steps, rotated-kernel option, pointing (radians),
    // per-visibility hour angles (device pointer once the call has staged
    // them) and the beam's spherical-harmonic coefficients (host)
    int ntimesteps = 0, aproj_opt = 0;
    double obs_dec = 0.0, obs_ra = 0.0;
    const double* lha = nullptr;
    const double* pbcoefs = nullptr;
    int npbcoefs = 0;
    // compensated FP32 only: grid cells stored in double and the c2r done in
    // double precision (wide_fft_needed decides)
    int wide_fft = 0;
    int own_c2r = 0; // the c2r on our own kernels (own_c2r_applies decides)
};

// W-projection with a maximum support above 32: the W-kernel tables are sized
// from the measured plane supports (a host round trip) instead of from the
// worst case, so such calls are not captured into CUDA graphs.
bool large_support(const ImagerSetup& s) { return s.nplanes > 0 && s.max_support > 32; }

// Sizes of the W-kernel generation (WideFieldImaging, aw_projection.cpp:19-111).
struct WkShape {
    int64_t workarea = 2, arr = 0;
    int half = 0, lh = 0;
    int ctas = 1;                              // CTAs that share a plane in k_wkernel_plane
    int smem_ctab = 0, smem_Q = 0, smem_T = 0; // what its shared memory holds
    size_t smem = 0;
    size_t q_cells = 0, t_cells = 0; // scratch for what it does not hold

    bool too_large() const { return arr > 46340; } // arr^2 > 2^31: not generated
};

WkShape wk_shape(const ImagerSetup& s, int os)
{
    WkShape k;
    const int K = 2 * s.max_support + 1;
    const int u = s.undersampling > 0 ? int(std::pow(2, s.undersampling - 1)) : 0;
    if (u > 0) {
        while (k.workarea / u < K)
            k.workarea *= 2;
    } else {
        while (k.workarea < s.N)
            k.workarea *= 2;
    }
    k.arr = k.workarea * os;
    if (k.too_large())
        return k;
    k.half = int(k.workarea / 2);
    k.lh = int(std::min<int64_t>(int64_t(s.max_support) * os + os / 2 + 1, k.arr / 2 + 1));
    // by the kernel's rows at the largest support (a second CTA costs little
    // where the truncated kernel turns out small), as far as the planes leave SMs
    k.ctas = std::max(1, std::min({ 4, k.lh / 16, 148 / std::max(s.nplanes, 1) }));
    // shared memory: the cosine table, Q and T in this order of preference (a
    // kernel of 16 cells' support and oversampling 8 on four CTAs takes 4 + 16
    // + 17 KB)
    auto fits = [&](size_t bytes) {
        if (k.smem + bytes > 160 * 1024)
            return 0;
        k.smem += bytes;
        return 1;
    };
    const size_t t_rows = size_t(ceil_div(k.lh, k.ctas));
    k.smem_ctab = fits(pad16(sizeof(double) * size_t(k.arr)));
    k.smem_Q = fits(sizeof(double2) * size_t(k.half) * k.half);
    k.smem_T = fits(sizeof(double2) * t_rows * k.half);
    if (!s.hankel && s.ntimesteps == 0) {
        k.q_cells = k.smem_Q ? 0 : size_t(s.nplanes) * k.half * k.half;
        k.t_cells = k.smem_T ? 0 : size_t(s.nplanes) * k.ctas * t_rows * k.half;
    }
    return k;
}

void check_pars(const ImagerSetup& s)
{
    if (s.N <= 0 || (s.N % 2) != 0)
        fail(STPGPU_ERR_INVALID_ARG, "grid size must be a positive even number");
    if (s.support <= 0)
        fail(STPGPU_ERR_INVALID_ARG, "kernel_support must be > 0");
    if (s.nplanes > 0 && s.max_support <= 0)
        fail(STPGPU_ERR_INVALID_ARG, "max_wpconv_support must be > 0 with W-projection");
    if (s.nplanes > 65535)
        fail(STPGPU_ERR_INVALID_ARG, "num_wplanes too large");
    if (s.nplanes > 0 && s.max_support > 127)
        fail(STPGPU_ERR_UNSUPPORTED, "max_wpconv_support > 127 is outside the GPU path");
    if (s.nplanes == 0 && s.support > 32)
        fail(STPGPU_ERR_UNSUPPORTED, "kernel_support > 32 is outside the GPU path");
    if (s.os > 4096)
        fail(STPGPU_ERR_INVALID_ARG, "oversampling too large");
}

// Size class of a call: those whose data could not take the W-planes without
// the |w| sort are remembered by it.
std::string size_class(const ImagerSetup& s, int precision)
{
    const int conv = s.nplanes > 0 ? s.max_support : s.support;
    // W-projection: the truncation percentage decides the plane supports, so it is part of the class
    return "p" + std::to_string(precision) + "/k" + std::to_string(s.nplanes > 0 ? 2 : (s.kernel_exact ? 1 : 0))
        + "/N" + std::to_string(s.N) + "/S" + std::to_string(conv) + "/os" + std::to_string(s.os)
        + (s.nplanes > 0 ? "/t" + fkey(s.trunc_perc) : std::string());
}

// Entries that n visibilities can have: two copies (original, mirrored) of up
// to two columns; more wraps only on grids smaller than two footprints.
uint64_t entry_capacity(int N, int K, int64_t n)
{
    return uint64_t(std::max<int64_t>(n, 1)) * (N >= 2 * K + 2 ? 4 : 18);
}

// The bins of a call's entries; the count, off, cursor and rank buffers are
// sized here and the flags attached.
BlockBins make_bins(stpgpu_context* c, const ImagerSetup& s, const GridOut& g, int64_t n, bool exact)
{
    BlockBins b {};
    const int K = 2 * (s.nplanes > 0 ? s.max_support : s.support) + 1;
    b.N = s.N;
    b.rows = g.image_rows;
    b.pad = int(ceil_div(K - 1, kBlk));
    b.brn = int(ceil_div(b.rows, kBlk)) + b.pad;
    b.bcn = int(ceil_div(b.N, kBlk)) + b.pad;
    b.wrap_neg = exact;
    b.support = s.support;
    b.ntimesteps = std::max(s.ntimesteps, 1);
    b.n = n;
    const size_t nbins = size_t(b.brn) * size_t(b.bcn);
    b.off = c->buf<uint32_t>("toff", nbins + size_t(b.bcn));
    b.count = c->buf<uint32_t>("tcount", nbins);
    b.cursor = c->buf<uint32_t>("tcur", nbins);
    b.ranks = c->buf<uint32_t>("tranks", size_t(std::max<int64_t>(n, 1)) * kEntrySlots);
    b.rank_overflow = g.d_err + CF_RANK_OVERFLOW;
    return b;
}

// Visibilities per block of cells above which several warps share a block.  On
// a small grid a warp a block leaves most of the GPU idle, and a block of a
// concentrated coverage keeps the rest waiting; on a large one there are warps
// enough, and a CTA that stages its entries once spends less on them.  The
// host knows neither the coverage nor the fullest block, so the line lies
// between the two: kernel, a warp a block and eight, us, disk / normal / tracks
// coverage at 24.5, 40 and 80 visibilities a block, W-kernels (support 2 to 3)
// in compensated single precision:
//   512^2   25 31, 41 34, 111 47 / 116 46, 174 60, 324 106 / 129 40, 140 53, 256 86
//   1500^2  64 178, 120 201, 286 292 / 182 156, 272 206, 527 335 / 186 151, 250 198, 455 325
//   2048^2  105 320, 198 358, 480 533 / 225 266, 355 353, 688 578 / 221 258, 336 339, 609 560
//   3000^2  205 673, 395 760, 947 1123 / 365 541, 560 718, 1062 1162 / 373 520, 573 684, 1095 1110
//   4096^2  368 1256, 716 1409 at 24.5 and 40 / 592 992, 910 1313 / 627 947, 938 1251
// and separable kernels on 2048^2 72 118, 111 149, 216 232 / 142 127, 168 162,
// 330 254 / 123 120, 155 154, 309 245.  With a beam in single precision (two
// CTAs an SM) 299 370 and 770 562 at 40 and 80 on 2048^2 / 435 372, 851 601.
constexpr int kDenseSplit = 8;
int64_t dense_per_block(int64_t blocks, bool beam, bool single)
{
    return blocks <= 20000 ? 24 : blocks / (beam && single ? 980 : 490);
}
// Columns of blocks that a CTA takes on sparse grids (k_grid_blocks).
constexpr int kSparseCols = 8;

// Where a call's items and kernel tables are, for grid_blocks.
template <typename R>
struct GridInputs {
    bool wproj = false, exact = false;
    int os = 1, cs = 1;
    const Item<R>* items = nullptr;
    // W-projection: planes (k_wsel_* or the sorting path) and kernels
    const int* plane_support = nullptr;
    const uint16_t* plane16 = nullptr;
    const uint32_t* order = nullptr;
    const int64_t* first = nullptr;
    int P = 0;
    const uint8_t* ts_of = nullptr;
    const uint32_t* wk_off = nullptr;
    const void* wk = nullptr;
    const unsigned int* max_support = nullptr;
    // separable kernels: 1-D table; exact: fractional positions
    const double* k1d = nullptr;
    const double* frac = nullptr;
};

// Binning by first cell and the block gridder (gridder_kernels.cuh).  wide:
// a single-precision call's grid holds double cells.
template <typename R, typename T, typename ACC>
void grid_blocks(stpgpu_context* c, const ImagerSetup& s, GridOut& g, int64_t n, BlockBins b, const GridInputs<R>& in,
    bool wide)
{
    cudaStream_t st = c->stream;
    const int K = 2 * (in.wproj ? s.max_support : s.support) + 1;
    const int64_t nn = std::max<int64_t>(n, 1);
    b.plane_support = in.plane_support;
    b.plane16 = in.plane16;
    b.order = in.order;
    b.first = in.first;
    b.P = in.P;
    b.ts_of = in.ts_of;
    const uint64_t cap = entry_capacity(s.N, K, nn);
    if (cap > 0xffffffffull)
        fail(STPGPU_ERR_INVALID_ARG, "too many visibilities for one snapshot");
    BinFill<R> q {};
    q.rec = c->buf<GridRec<R>>("trecs", cap);
    q.wts = s.beam ? c->buf<R>("trecw", cap) : nullptr;
    q.cap = cap;
    q.wk_off = in.wk_off;
    q.cs = in.cs;
    q.os = in.os;
    q.exact = in.exact;
    q.err = g.d_err;
    if (n > 0 && in.wproj) {
        k_bin_count<R><<<grid1d(n, 256), 256, 0, st>>>(b, in.items);
        STPGPU_CHECK_LAUNCH();
    }
    g.d_nitems = g.d_err + CF_ENTRIES;
    k_bin_scan<<<unsigned(b.bcn), 256, 0, st>>>(b.count, const_cast<uint32_t*>(b.off), b.cursor, b.brn, b.rank_overflow,
        g.d_nitems);
    STPGPU_CHECK_LAUNCH();
    if (n > 0) {
        k_bin_fill<R><<<grid1d(n, 256), 256, 0, st>>>(b, in.items, q);
        STPGPU_CHECK_LAUNCH();
    }
    // columns that start on a 128-byte line where our own kernels read them
    g.ld = s.own_c2r ? int(ceil_div(b.rows, 16)) * 16 : b.rows;
    const size_t cells = size_t(g.ld) * b.N;
    const bool f64 = sizeof(R) == 8 || wide;
    g.grid = c->buf<unsigned char>("grid", cells * (f64 ? 16 : 8));
    g.beam = s.beam ? c->buf<unsigned char>("beamgrid", cells * (f64 ? 16 : 8)) : nullptr;
    auto geometry = [&](auto& p) {
        p.N = b.N;
        p.rows = b.rows;
        p.pad = b.pad;
        p.brn = b.brn;
        p.ld = g.ld;
        p.off = b.off;
        p.recs = q.rec;
        p.wts = q.wts;
        p.grid = g.grid;
        p.beam = g.beam;
    };
    const int64_t nbr = ceil_div(b.rows, kBlk), nbc = ceil_div(b.N, kBlk);
    const bool dense = n > dense_per_block(nbr * nbc, s.beam, sizeof(T) == 4) * nbr * nbc;
    const unsigned nbr8 = unsigned(ceil_div(nbr, kGridWarps));
    // Few visibilities: several columns of blocks a CTA, as long as the CTAs
    // still fill the GPU.  One column and eight, us, at disk / normal coverage,
    // separable kernels in single precision, then W-kernels in double: 4096^2
    // (2112 CTAs of eight columns) at 0.3, 0.5 and 1 visibility a block 56 32,
    // 56 34, 60 36 / 44 33, 46 37, 50 48, then 74 53, 77 57, 84 65 / 59 62, 63
    // 72, 72 98; 5000^2 (3120) at 1 and 2 85 47, 93 68 / 71 60, 84 88, then 126
    // 87, 143 131 / 108 129, 132 158; 6000^2 (4418) at 1, 2 and 3 124 63, 133
    // 88, 142 109 / 103 74, 120 107, 139 157, then 180 122, 207 183, 235 227 /
    // 154 166, 189 209, 224 263; 8192^2 at 2 and 3 248 160, 266 199 / 219 174,
    // 251 236, then 390 333, 446 422 / 350 332, 418 423.
    const int64_t ctas = nbr8 * (nbc / kSparseCols);
    const double line = ctas < 148 * 4 ? 0.0 : (ctas < 148 * 20 ? 0.5 : (ctas < 4000 ? 1.5 : 2.0));
    const bool sparse = double(n) < line * double(nbr * nbc);
    auto run = [&](auto core, const auto& p) {
        using C = decltype(core);
        c->mark(1);
        if (dense)
            k_grid_dense<C, kDenseSplit><<<dim3(unsigned(ceil_div(nbr, kGridWarps / kDenseSplit)), unsigned(nbc)),
                32 * kGridWarps, 0, st>>>(p);
        else
            sparse ? k_grid_blocks<C, kSparseCols><<<dim3(nbr8, unsigned(ceil_div(nbc, kSparseCols))), 32 * kGridWarps, 0, st>>>(p)
                   : k_grid_blocks<C, 1><<<dim3(nbr8, unsigned(nbc)), 32 * kGridWarps, 0, st>>>(p);
        STPGPU_CHECK_LAUNCH();
        c->mark(2);
    };
    auto by_cell = [&](auto f) { // f(the grid's scalar type)
        if constexpr (sizeof(R) == 8)
            f(double());
        else
            f64 ? f(double()) : f(float());
    };
    if (in.wproj) {
        WprojParams<R, T> p {};
        geometry(p);
        p.wk = static_cast<const typename Cplx<T>::T*>(in.wk);
        p.max_support = in.max_support;
        by_cell([&](auto cell) {
            using G = decltype(cell);
            s.beam ? run(WprojCore<R, G, T, ACC, true>(), p) : run(WprojCore<R, G, T, ACC, false>(), p);
        });
        return;
    }
    SepParams<R> p {};
    geometry(p);
    p.K = K;
    if (in.exact) {
        double* tab = c->buf<double>("exact_tab", size_t(nn) * 2 * K);
        if (n > 0) {
            k_exact_tables<<<grid1d(2 * n, 256), 256, 0, st>>>(s.kf, s.trunc, s.support, in.frac, n, tab);
            STPGPU_CHECK_LAUNCH();
        }
        p.tab = tab;
    } else {
        p.tw = kBlk * b.pad + 15;
        p.zrow = in.cs * p.tw;
        double* tab = c->buf<double>("k1dpad", size_t(in.cs + 1) * p.tw);
        if (!c->memo("k1dpad", std::to_string(s.kf) + "/" + fkey(s.trunc) + "/" + std::to_string(s.support) + "/"
                    + std::to_string(in.os))) {
            k_pad_table<<<grid1d(int64_t(in.cs + 1) * p.tw, 256), 256, 0, st>>>(in.k1d, in.cs, K, p.tw, tab);
            STPGPU_CHECK_LAUNCH();
        }
        p.tab = tab;
    }
    by_cell([&](auto cell) {
        using G = decltype(cell);
        if (in.exact)
            s.beam ? run(SepCore<R, G, true, true, false>(), p) : run(SepCore<R, G, true, false, false>(), p);
        else if (p.zrow + p.tw <= SepCore<R, G, false, false, true>::kTab) // (oversampling 16 at support 4: 414 values)
            s.beam ? run(SepCore<R, G, false, true, true>(), p) : run(SepCore<R, G, false, false, true>(), p);
        else
            s.beam ? run(SepCore<R, G, false, true, false>(), p) : run(SepCore<R, G, false, false, false>(), p);
    });
}

// convolve_to_grid (gridder.h:240-997): grids into context buffers "grid"
// and "beamgrid" of precision R (complex), image_rows x N column-major.
template <typename R, int COMP>
GridOut run_gridder(stpgpu_context* c, const ImagerSetup& s, const void* d_vis, int vis_c64, const double* d_wts,
    const double* d_uv, int uv_is_pixels, int64_t n)
{
    // W-projection: kernel tables in the call's precision, sums in double except for plain FP32
    using KT = R;
    using ACC = std::conditional_t<sizeof(R) == 8 || COMP == 1, double, float>;
    using C2 = typename Cplx<KT>::T;
    check_pars(s);
    cudaStream_t st = c->stream;
    GridOut g;
    const int N = s.N;
    const bool wproj = s.nplanes > 0;
    const int conv_support = wproj ? s.max_support : s.support;
    const int kernel_exact = wproj ? 0 : s.kernel_exact;
    int os = s.os;
    if (kernel_exact) {
        os = 1;
    } else {
        os = (os >> 1) << 1;
        if (os == 0)
            os = 1;
    }
    const int cs = (os / 2) * 2 + 1;
    const int image_rows = s.halfplane ? N / 2 + 1 : N;
    g.image_rows = image_rows;
    const int64_t nn = std::max<int64_t>(n, 1);
    c->mark(0);

    // ---- prepass (gridder.h:369-423, :504)
    Item<R>* items = c->buf<Item<R>>("items", nn);
    const unsigned nb_pre = std::min<unsigned>(grid1d(n, GRID_THREADS), 148 * 8);
    double* wpart = c->buf<double>("wpart", nb_pre);
    unsigned long long* npart = c->buf<unsigned long long>("npart", nb_pre);
    g.d_total = c->buf<double>("total", 4);
    g.d_ngood = c->buf<unsigned long long>("ngood", 2);
    g.d_err = c->buf<unsigned int>("err", CF_WORDS);
    BlockBins bins = make_bins(c, s, g, n, kernel_exact != 0);
    const bool use_wsel = wproj && n > 0 && s.wsel;
    int wsel_log = WSEL_MIN_LOG;
    while (wsel_log < WSEL_MAX_LOG && (int64_t(8) << wsel_log) < n)
        wsel_log++;
    WselState* ws = use_wsel ? c->buf<WselState>("wsel", 1) : nullptr;
    zero_words(st, { { g.d_err, CF_WORDS }, { bins.count, int64_t(bins.brn) * bins.bcn },
                       { ws, use_wsel ? int64_t(1) << wsel_log : 0 },
                       { ws ? ws->cursor : nullptr, use_wsel ? int64_t(kWselZeroWords) : 0 } });
    PrepassParams pp {};
    pp.n = n;
    pp.vis = d_vis;
    pp.vis_c64 = vis_c64;
    pp.weights = d_wts;
    pp.uv = d_uv;
    pp.uv_is_pixels = uv_is_pixels;
    pp.inv_px = arc_sec_to_rad(s.cell_size) * double(N); // imager.h:293
    pp.N = N;
    pp.conv_support = conv_support;
    pp.halfplane = s.halfplane;
    pp.shift_uv = s.shift_uv;
    pp.kernel_exact = kernel_exact;
    pp.os = os;
    pp.keep_w = wproj ? 1 : 0;
    pp.frac = kernel_exact ? c->buf<double>("frac", 2 * nn) : nullptr;
    pp.wsum_part = wpart;
    pp.ngood_part = npart;
    pp.absw_key = wproj ? c->buf<double>("absw", nn) : nullptr;
    pp.wmax_part = (wproj && !s.full_wsort) ? c->buf<double>("wmaxpart", 2 * size_t(nb_pre)) : nullptr;
    pp.iota = (wproj && !s.wsel) ? c->buf<uint32_t>("perm_in", nn) : nullptr;
    pp.ticket = g.d_err + CF_TICKET;
    pp.total = g.d_total;
    pp.ngood = g.d_ngood;
    if (wproj)
        bins.count = nullptr; // (counted once the supports are known)
    k_prepass<R><<<nb_pre, GRID_THREADS, 0, st>>>(pp, items, bins); // n = 0 too: one block, totals of zero
    STPGPU_CHECK_LAUNCH();
    if (wproj)
        bins.count = c->buf<uint32_t>("tcount", 1);

    // ---- kernels
    const uint32_t* sorted_perm = nullptr;
    Item<R>* items_sorted = nullptr; // W-projection: the items in |w| order
    const int64_t* plane_first = nullptr;
    int nplanes = 0;
    const double* k1d64 = nullptr;
    C2* wk = nullptr;
    uint32_t* wk_off = nullptr;
    uint8_t* ts_of = nullptr; // A-projection time step per visibility
    int* plane_support = nullptr;
    if (!wproj && !kernel_exact) {
        // populate_kernel_cache (gridder.h:73-105) as a 1-D table, FP64 on the device
        const int K = 2 * s.support + 1;
        const std::string key = std::to_string(s.kf) + "/" + fkey(s.trunc) + "/" + std::to_string(s.support)
            + "/" + std::to_string(os);
        double* t64 = c->buf<double>("k1d64", size_t(cs) * K);
        if (!c->memo("k1d64", key)) {
            k_kernel_table<<<grid1d(cs, 64), 64, 0, st>>>(s.kf, s.trunc, s.support, os, t64);
            STPGPU_CHECK_LAUNCH();
        }
        k1d64 = t64;
    }
    const uint16_t* plane16 = nullptr;
    if (use_wsel) {
        // the planes without sorting (k_wsel_*, see imager_kernels.cuh); a
        // condition it cannot meet sets error bit 16 and the caller grids
        // again on the sorting path
        const int P = s.nplanes;
        const unsigned g2 = std::min<unsigned>(grid1d(n, 256), 148 * 8);
        k_wsel_hist<<<std::min<unsigned>(grid1d(n, 1024), 148), 1024, 0, st>>>(pp.absw_key, n, g.d_total, ws, wsel_log, P,
            g.d_ngood, g.d_err);
        STPGPU_CHECK_LAUNCH();
        // members of the start bins: at most P - 1 bins of WSEL_CAP
        unsigned long long* mbits = c->buf<unsigned long long>("wsel_mb", size_t(std::max(P - 1, 1)) * WSEL_CAP);
        uint32_t* midx = c->buf<uint32_t>("wsel_mi", size_t(std::max(P - 1, 1)) * WSEL_CAP);
        k_wsel_collect<<<g2, 256, 0, st>>>(pp.absw_key, n, g.d_total, ws, wsel_log, mbits, midx);
        STPGPU_CHECK_LAUNCH();
        if (P > 1) {
            k_wsel_resolve<<<P - 1, 256, 0, st>>>(ws, mbits, midx);
            STPGPU_CHECK_LAUNCH();
        }
        uint16_t* pl = c->buf<uint16_t>("wsel_plane", nn);
        int64_t* first = c->buf<int64_t>("pfirst", P);
        double* w_avg = c->buf<double>("wavg", P);
        k_wsel_classify<<<g2, 256, 0, st>>>(pp.absw_key, n, P, g.d_total, ws, pl, g.d_err, w_avg, first);
        STPGPU_CHECK_LAUNCH();
        plane16 = pl;
        plane_first = first;
        nplanes = P;
    } else if (wproj && n > 0) {
        const int P = s.nplanes;
        // |w| order (gridder.h:311-367): stable radix sort of 24-bit keys of
        // |w| (k_wkey24; three digit passes instead of the eight of the 64-bit
        // sort), then runs of equal keys re-sorted by the full |w| bits; with
        // full_wsort the IEEE bits of |w| themselves are sorted (64-bit keys;
        // non-negative doubles order as their bit patterns).
        const unsigned long long* keys64 = reinterpret_cast<const unsigned long long*>(pp.absw_key);
        uint32_t* perm_in = pp.iota;
        uint32_t* perm = c->buf<uint32_t>("perm", nn);
        size_t tb = 0;
        if (s.full_wsort) {
            unsigned long long* k64out = c->buf<unsigned long long>("absw64_sorted", nn);
            cub::DeviceRadixSort::SortPairs(nullptr, tb, keys64, k64out, perm_in, perm, int(n), 0, 64, st);
            void* tmp = c->buf<unsigned char>("cubtmp", tb);
            if (cub::DeviceRadixSort::SortPairs(tmp, tb, keys64, k64out, perm_in, perm, int(n), 0, 64, st)
                != cudaSuccess)
                fail(STPGPU_ERR_CUDA, "radix sort failed");
        } else {
            uint32_t* key24 = c->buf<uint32_t>("absw24", nn);
            k_wkey24<<<std::min<unsigned>(grid1d(n, 256), 148 * 8), 256, 0, st>>>(pp.absw_key, n, g.d_total, key24);
            STPGPU_CHECK_LAUNCH();
            uint32_t* k32out = c->buf<uint32_t>("absw24_sorted", nn);
            cub::DeviceRadixSort::SortPairs(nullptr, tb, key24, k32out, perm_in, perm, int(n), 0, 24, st);
            void* tmp = c->buf<unsigned char>("cubtmp", tb);
            if (cub::DeviceRadixSort::SortPairs(tmp, tb, key24, k32out, perm_in, perm, int(n), 0, 24, st)
                != cudaSuccess)
                fail(STPGPU_ERR_CUDA, "radix sort failed");
            k_fix_runs<<<grid1d(n, 256), 256, 0, st>>>(k32out, perm, keys64, n, g.d_err);
            STPGPU_CHECK_LAUNCH();
        }
        uint8_t* good_sorted = c->buf<uint8_t>("good_sorted", nn);
        uint32_t* gflag = c->buf<uint32_t>("gflag", nn + 1);
        uint32_t* cgood = c->buf<uint32_t>("cgood", nn + 1);
        double* absw_sorted = c->buf<double>("absw_sorted", nn);
        // binning and gridding read the items in |w| order (sequential
        // passes instead of gathers through the permutation)
        items_sorted = c->buf<Item<R>>("items_sorted", nn);
        k_gather_good<R><<<grid1d(n, 256), 256, 0, st>>>(perm, items, pp.absw_key, n, good_sorted, gflag, absw_sorted,
            items_sorted);
        STPGPU_CHECK_LAUNCH();
        zero_words(st, { { gflag + n, 1 } });
        size_t tb2 = 0;
        cub::DeviceScan::ExclusiveSum(nullptr, tb2, gflag, cgood, int(n + 1), st);
        void* tmp2 = c->buf<unsigned char>("cubtmp2", tb2);
        if (cub::DeviceScan::ExclusiveSum(tmp2, tb2, gflag, cgood, int(n + 1), st) != cudaSuccess)
            fail(STPGPU_ERR_CUDA, "scan failed");
        int64_t* first = c->buf<int64_t>("pfirst", P);
        int64_t* last = c->buf<int64_t>("plast", P);
        double* w_avg = c->buf<double>("wavg", P);
        k_wplanes<<<std::min<unsigned>(grid1d(n, 256), 148 * 4), 256, 0, st>>>(cgood, n, P, c->buf<uint32_t>("goodpos", nn),
            g.d_err + CF_TICKET, first, last);
        STPGPU_CHECK_LAUNCH();
        if (s.wmedian) {
            k_wplane_values<<<P, 256, 0, st>>>(cgood, absw_sorted, good_sorted, first, last, n, P, 1, w_avg);
            STPGPU_CHECK_LAUNCH();
        } else {
            const int nblk = int(std::min<int64_t>(2048, ceil_div(n, 512)));
            const int64_t chunk = ceil_div(n, nblk);
            double* partial = c->buf<double>("wpartial", size_t(P) * nblk);
            k_wplane_partial<<<nblk, 256, 0, st>>>(absw_sorted, good_sorted, first, last, n, P, chunk, nblk, partial);
            STPGPU_CHECK_LAUNCH();
            k_wplane_finish<<<P, 256, 0, st>>>(partial, cgood, first, last, chunk, nblk, w_avg);
            STPGPU_CHECK_LAUNCH();
        }
        sorted_perm = perm;
        plane_first = first;
        nplanes = P;
    }
    if (wproj && n > 0) {
        const int P = s.nplanes;
        double* w_avg = c->buf<double>("wavg", P); // the plane means, from either path above
        // W-kernels in FP64 (WideFieldImaging, aw_projection.cpp:19-111,173-210,366-452)
        const int K = 2 * s.max_support + 1;
        const WkShape ks = wk_shape(s, os);
        if (ks.workarea < K)
            fail(STPGPU_ERR_INVALID_ARG, "W-kernel workarea smaller than the kernel size");
        if (ks.arr % 2)
            fail(STPGPU_ERR_INVALID_ARG, "array_size must be multiple of 2 for WideFieldImaging generation.");
        if (ks.too_large())
            fail(STPGPU_ERR_UNSUPPORTED, "W-kernel array too large");
        const int workarea = int(ks.workarea), arr = int(ks.arr), half = ks.half, Lh = ks.lh;
        const double scaling = double(N) / double(workarea);
        double* aa = c->buf<double>("aa", workarea);
        if (!c->memo("aa", std::to_string(s.kf) + "/" + fkey(s.trunc) + "/" + std::to_string(workarea) + "/"
                               + std::to_string(s.analytic))) {
            // ImgDomKernel(kernel_creator, workarea) (gridder.h:486)
            const int centre = workarea / 2;
            const int dmax = int(std::floor(s.trunc)) + 1;
            double ssum = 0.0;
            for (int d = -std::min(dmax, centre); d <= std::min(dmax, workarea - centre - 1); d++)
                ssum += kernel_value(s.kf, s.trunc, double(d));
            const double ksum_inv = ssum > 0.0 ? 1.0 / ssum : 1.0;
            k_imgdom_kernel<<<grid1d(workarea, 128), 128, 0, st>>>(s.kf, s.trunc, workarea, s.analytic, ksum_inv,
                dmax, aa);
            STPGPU_CHECK_LAUNCH();
        }
        double* ctab = c->buf<double>("ctab", arr);
        if (!c->memo("ctab", std::to_string(arr))) {
            k_cos_table<<<grid1d(arr, 256), 256, 0, st>>>(arr, ctab);
            STPGPU_CHECK_LAUNCH();
        }
        WkParams wq {};
        wq.w_avg = w_avg;
        wq.aa = aa;
        wq.ctab = ctab;
        wq.half = half;
        wq.arr = arr;
        wq.os = os;
        wq.cs = cs;
        wq.max_support = s.max_support;
        wq.lh_max = Lh;
        // WideFieldImaging gets real_t(arc_sec_to_rad(cell)), scaled by N/workarea
        wq.scaled_cell = arc_sec_to_rad(s.cell_size) * scaling;
        wq.trunc_perc = s.trunc_perc;
        wq.smem_ctab = ks.smem_ctab;
        wq.smem_Q = ks.smem_Q;
        wq.smem_T = ks.smem_T;
        wq.Qs = ks.q_cells ? c->buf<double2>("wkQ", ks.q_cells) : nullptr;
        wq.Ts = ks.t_cells ? c->buf<double2>("wkT", ks.t_cells) : nullptr;
        wq.convd = c->buf<double2>("wkconv", size_t(P) * Lh * Lh);
        const int T = std::max(s.ntimesteps, 1);
        const int PT = P * T;
        plane_support = c->buf<int>("psupport", PT);
        wq.support = plane_support;
        const double2* aconv = nullptr; // A-projection: transformed kernels [P*T][arr][arr]
        if (s.ntimesteps > 0) {
            // time steps and their parallactic angles (gridder.h:507-520, gridder.cpp:148-200)
            double* iv = c->buf<double>("ap_iv", T + 1);
            double* lmean = c->buf<double>("ap_lmean", T);
            double* angle = c->buf<double>("ap_angle", T);
            ts_of = c->buf<uint8_t>("ap_ts", nn);
            k_lha_intervals<<<1, 1024, 0, st>>>(s.lha, n, T, iv);
            STPGPU_CHECK_LAUNCH();
            k_lha_steps<R><<<grid1d(n, 256), 256, 0, st>>>(s.lha, items, n, T, iv, ts_of);
            STPGPU_CHECK_LAUNCH();
            k_lha_means<R><<<T, 256, 0, st>>>(s.lha, items, ts_of, n, lmean);
            STPGPU_CHECK_LAUNCH();
            k_parangle<<<1, 256, 0, st>>>(lmean, T, s.obs_dec, s.obs_ra, angle);
            STPGPU_CHECK_LAUNCH();
            // inverse primary beam per step (one unrotated beam with aproj_opt)
            double* coefs = c->buf<double>("ap_coefs", s.npbcoefs);
            STPGPU_CUDA_TRY(
                cudaMemcpyAsync(coefs, s.pbcoefs, sizeof(double) * s.npbcoefs, cudaMemcpyHostToDevice, st));
            const int deg = (s.npbcoefs - 1) / 2;
            const double fov = arc_sec_to_rad(s.cell_size) * double(N);
            const int nA = s.aproj_opt ? 1 : T;
            double* Abeam = c->buf<double>("ap_beam", size_t(nA) * workarea * workarea);
            k_aproj_beam<<<grid1d(int64_t(nA) * workarea * workarea, 256), 256, 0, st>>>(nA, workarea, fov, coefs, deg,
                s.aproj_opt ? nullptr : angle, Abeam);
            STPGPU_CHECK_LAUNCH();
            // W-screen x beam, 2-D FFT per (plane, step) or per plane
            const int G = P * nA;
            const size_t img = size_t(arr) * arr;
            const size_t nimg = size_t(G) + (s.aproj_opt ? size_t(PT) : 0);
            if (nimg * img * sizeof(double2) > (uint64_t(8) << 30))
                fail(STPGPU_ERR_UNSUPPORTED,
                    "A-projection kernels exceed 8 GB (planes x time steps x (workarea x oversampling)^2)");
            double2* abuf = c->buf<double2>("ap_fft", nimg * img);
            STPGPU_CUDA_TRY(cudaMemsetAsync(abuf, 0, sizeof(double2) * size_t(G) * img, st));
            const int span = 2 * half - 1;
            k_aproj_screen<<<grid1d(int64_t(G) * span * span, 256), 256, 0, st>>>(wq, P, nA, Abeam, abuf);
            STPGPU_CHECK_LAUNCH();
            if (cufftExecZ2Z(c->plan_many(arr, CUFFT_Z2Z, G), reinterpret_cast<cufftDoubleComplex*>(abuf),
                    reinterpret_cast<cufftDoubleComplex*>(abuf), CUFFT_FORWARD)
                != CUFFT_SUCCESS)
                fail(STPGPU_ERR_CUFFT, "A-projection kernel FFT failed");
            k_aproj_support<<<grid1d(G, 128), 128, 0, st>>>(abuf, G, arr, os, s.max_support, s.trunc_perc,
                s.aproj_opt ? T : 1, plane_support);
            STPGPU_CHECK_LAUNCH();
            aconv = abuf;
            if (s.aproj_opt) {
                // rotate each plane's kernel by the step's angle, step after
                // step on the previous step's result (gridder.h:732-737)
                double2* rot = abuf + size_t(G) * img; // [P][T][arr][arr]
                for (int t = 0; t < T; t++) {
                    const double2* src = t == 0 ? abuf : rot + size_t(t - 1) * img;
                    const int64_t src_stride = t == 0 ? int64_t(img) : int64_t(T) * int64_t(img);
                    k_aproj_rotate<<<grid1d(int64_t(P) * int64_t(img), 256), 256, 0, st>>>(src, src_stride,
                        rot + size_t(t) * img, int64_t(T) * int64_t(img), P, arr, angle, t);
                    STPGPU_CHECK_LAUNCH();
                }
                aconv = rot;
            }
        } else if (s.hankel) {
            HankelParams hq {};
            hq.n = s.proj_slice ? arr : arr / 2;
            if (hq.n < 3)
                fail(STPGPU_ERR_INVALID_ARG, "Hankel transform needs more than 2 radial samples");
            hq.proj_slice = s.proj_slice;
            hq.cubic = s.cubic;
            hq.R = c->buf<double2>("hkR", size_t(P) * half);
            hq.Y = c->buf<double2>("hkY", size_t(P) * hq.n);
            hq.B = c->buf<double2>("hkB", size_t(P) * hq.n);
            hq.Cp = c->buf<double>("hkC", size_t(P) * 2 * hq.n);
            k_hankel_plane<<<P, 1024, 0, st>>>(wq, hq);
        } else {
            if (ks.q_cells) {
                k_wk_quadrant<<<dim3(grid1d(int64_t(half) * half, 256), P), 256, 0, st>>>(wq);
                STPGPU_CHECK_LAUNCH();
            }
            STPGPU_CUDA_TRY(cudaFuncSetAttribute(k_wkernel_plane, cudaFuncAttributeMaxDynamicSharedMemorySize, 160 * 1024));
            k_wkernel_plane<<<dim3(P, ks.ctas), 1024, ks.smem, st>>>(wq);
        }
        STPGPU_CHECK_LAUNCH();
        // per-offset K x K tables in the gridder's precision: worst-case
        // capacity (every plane at the maximum support), or with large
        // supports the sum over the measured plane supports
        uint64_t cap_wk = uint64_t(PT) * cs * cs * uint64_t(K) * K;
        if (large_support(s)) {
            std::vector<int> sup(PT);
            STPGPU_CUDA_TRY(cudaMemcpyAsync(sup.data(), plane_support, sizeof(int) * PT, cudaMemcpyDeviceToHost, st));
            STPGPU_CUDA_TRY(cudaStreamSynchronize(st));
            cap_wk = 0;
            for (int v : sup)
                cap_wk += uint64_t(cs) * cs * uint64_t(2 * v + 1) * uint64_t(2 * v + 1);
            cap_wk = std::max<uint64_t>(cap_wk, 1);
        }
        if (cap_wk * sizeof(C2) > (uint64_t(16) << 30) || cap_wk > 0xffffffffull)
            fail(STPGPU_ERR_UNSUPPORTED, "W-kernel tables exceed 16 GB (planes x oversampling^2 x support^2)");
        wk = c->buf<C2>("wkexp", cap_wk);
        wk_off = c->buf<uint32_t>("wkoff", PT);
        if (aconv)
            k_aproj_expand<KT><<<dim3(PT, cs * cs), 256, 0, st>>>(aconv, arr, plane_support, cs, os, wk, wk_off,
                g.d_err + CF_MAX_SUPPORT);
        else
            k_wk_expand<KT><<<dim3(P, cs * cs), kExpandThreads, 0, st>>>(wq.convd, plane_support, P, cs, os, Lh,
                large_support(s) ? 0u : uint32_t(cs * cs) * uint32_t(K * K), wk, wk_off, g.d_err + CF_MAX_SUPPORT);
        STPGPU_CHECK_LAUNCH();
        g.d_plane_support = plane_support;
        g.nplanes = PT;
    }

    if (2 * conv_support + 1 > 255)
        fail(STPGPU_ERR_UNSUPPORTED, "kernel support > 127 is outside the GPU path");
    GridInputs<R> in;
    in.wproj = wproj;
    in.exact = kernel_exact != 0;
    in.os = os;
    in.cs = cs;
    in.items = items_sorted ? items_sorted : items;
    in.plane_support = plane_support;
    in.plane16 = plane16;
    in.order = sorted_perm;
    in.first = plane_first;
    in.P = nplanes;
    in.ts_of = ts_of;
    in.wk_off = wk_off;
    in.wk = wk;
    in.max_support = g.d_err + CF_MAX_SUPPORT;
    in.k1d = k1d64;
    in.frac = pp.frac;
    grid_blocks<R, KT, ACC>(c, s, g, n, bins, in, COMP == 1 && s.wide_fft);
    return g;
}

PackArgs pack_args(const GridOut& g, ScalarPack* out)
{
    return PackArgs { g.d_total, g.d_ngood, g.d_nitems, g.d_err, g.d_plane_support, g.nplanes, out };
}

// The call's scalars, once its kernels are done.  packed: the normalisation
// wrote them to the page-locked stage.
ScalarPack read_back(stpgpu_context* c, const GridOut& g, bool packed)
{
    ScalarPack* h = c->host_stage<ScalarPack>(1);
    if (!packed) {
        k_pack_scalars<<<1, 32, 0, c->stream>>>(pack_args(g, c->host_stage_dev(h)));
        STPGPU_CHECK_LAUNCH();
    }
    STPGPU_CUDA_TRY(cudaStreamSynchronize(c->stream));
    const ScalarPack r = *h;
    // bit 4: the 32-bit |w| sort met a long run of distinct |w| (the caller
    // repeats the gridding with the 64-bit sort); bit 16: the W-planes
    // without the sort did not apply (the caller grids again on the sorting
    // path); other bits are errors
    if (r.err & ~(4u | 16u))
        fail(STPGPU_ERR_DEVICE, "gridder reported internal error flags " + std::to_string(r.err));
    return r;
}

template <typename R>
const double* device_gcf(stpgpu_context* c, const ImagerSetup& s)
{
    double* gcf = c->buf<double>("gcf", s.N);
    c->buf<double>("gcfinv", s.N);
    if (c->memo("gcf", std::to_string(s.kf) + "/" + fkey(s.trunc) + "/" + std::to_string(s.N) + "/"
                          + std::to_string(s.analytic))
        && c->memo("gcfinv", std::to_string(s.kf) + "/" + fkey(s.trunc) + "/" + std::to_string(s.N) + "/"
            + std::to_string(s.analytic)))
        return gcf;
    c->memo("gcfinv", std::to_string(s.kf) + "/" + fkey(s.trunc) + "/" + std::to_string(s.N) + "/"
            + std::to_string(s.analytic));
    double ksum_inv = 1.0;
    const int dmax = int(std::floor(s.trunc)) + 1;
    if (!s.analytic) {
        const int centre = s.N / 2;
        double ssum = 0.0;
        for (int d = -std::min(dmax, centre); d <= std::min(dmax, s.N - centre - 1); d++)
            ssum += kernel_value(s.kf, s.trunc, double(d));
        ksum_inv = ssum > 0.0 ? 1.0 / ssum : 1.0;
    }
    k_imgdom_kernel<<<grid1d(s.N, 256), 256, 0, c->stream>>>(s.kf, s.trunc, s.N, s.analytic, ksum_inv, dmax, gcf);
    STPGPU_CHECK_LAUNCH();
    double* ginv = c->buf<double>("gcfinv", s.N);
    k_reciprocal<<<grid1d(s.N, 256), 256, 0, c->stream>>>(gcf, ginv, s.N);
    STPGPU_CHECK_LAUNCH();
    return gcf;
}

// Whether the c2r runs on our own kernels (k_fft_axis, k_c2r_normalise): grids
// of a power of two from 256 to 16384 in double and to 8192 in single precision
// (others take cuFFT's 2-D transform and k_normalise), an image that the kernel
// can store in pairs, and no single-precision transform into a double image.
// Transform and normalisation, cuFFT and ours: 8192^2 397 and 348 us in single,
// 866 and 644 in double precision; 16384^2 1512 and 1578 in single, 3616 and
// 2961 in double; 1024^2 26 and 24, 33 and 28.
bool own_c2r_applies(const ImagerSetup& s, bool fp64_fft, int out_f32, const void* image, const void* beam)
{
    const uintptr_t pair = out_f32 ? 8 : 16;
    return s.halfplane && (s.N & (s.N - 1)) == 0 && s.N >= (2 << kC2rMinLog)
        && s.N <= (2 << (fp64_fft ? kC2rMaxLog : kC2rMaxLogF))
        && (fp64_fft || out_f32) && reinterpret_cast<uintptr_t>(image) % pair == 0
        && reinterpret_cast<uintptr_t>(beam) % pair == 0;
}

// One pass of the columns-axis transform over transforms of length L.
template <typename T, bool FIRST>
void launch_axis(stpgpu_context* c, const GridOut& g, void* grid, int N, int L, const void* tw)
{
    using C = typename Cplx<T>::T;
    auto run = [&](auto len) {
        constexpr int l = decltype(len)::value;
        constexpr size_t smem = l > 16 ? size_t(axis_groups(l)) * l * 32 * sizeof(C) : 0;
        auto kern = k_fft_axis<T, l, FIRST>;
        if (smem > 48 * 1024)
            STPGPU_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)));
        const dim3 blocks(grid1d(g.image_rows, 32), unsigned(N / l / axis_groups(l)));
        kern<<<blocks, axis_threads(l), smem, c->stream>>>(static_cast<C*>(grid), g.ld, g.image_rows, N,
            static_cast<const C*>(tw));
        STPGPU_CHECK_LAUNCH();
    };
    switch (L) {
    case 16:
        return run(std::integral_constant<int, 16>());
    case 32:
        return run(std::integral_constant<int, 32>());
    case 64:
        return run(std::integral_constant<int, 64>());
    case 128:
        if constexpr (FIRST || sizeof(T) == 8) // (second pass: 16384 only)
            return run(std::integral_constant<int, 128>());
    }
    fail(STPGPU_ERR_UNSUPPORTED, "axis length");
}

template <typename T, typename RO, int LOGM>
void launch_c2r(stpgpu_context* c, const ImagerSetup& s, int image_size, int correction, const GridOut& g, const void* F,
    const void* tw, const double* ginv, void* out, ScalarPack* pack)
{
    using C = typename Cplx<T>::T;
    constexpr size_t smem = c2r_smem(LOGM, sizeof(C));
    auto kern = k_c2r_normalise<T, RO, LOGM>;
    if (smem > 48 * 1024)
        STPGPU_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)));
    kern<<<grid1d(image_size, c2r_rows(LOGM)), c2r_threads(LOGM), smem, c->stream>>>(static_cast<const C*>(F), g.ld,
        static_cast<const C*>(tw), image_size, g.d_total, ginv, correction, static_cast<RO*>(out), pack_args(g, pack));
    STPGPU_CHECK_LAUNCH();
}

template <typename T, typename RO>
void launch_c2r(stpgpu_context* c, const ImagerSetup& s, int image_size, int correction, const GridOut& g, const void* F,
    const void* tw, const double* ginv, void* out, ScalarPack* pack)
{
    auto run = [&](auto lm) {
        launch_c2r<T, RO, decltype(lm)::value>(c, s, image_size, correction, g, F, tw, ginv, out, pack);
    };
    switch (s.N) {
    case 256:
        return run(std::integral_constant<int, 7>());
    case 512:
        return run(std::integral_constant<int, 8>());
    case 1024:
        return run(std::integral_constant<int, 9>());
    case 2048:
        return run(std::integral_constant<int, 10>());
    case 4096:
        return run(std::integral_constant<int, 11>());
    case 8192:
        return run(std::integral_constant<int, 12>());
    case 16384:
        if constexpr (sizeof(T) == 8)
            return run(std::integral_constant<int, 13>());
    }
    fail(STPGPU_ERR_UNSUPPORTED, "c2r size");
}

template <typename R>
void finish_own(stpgpu_context* c, const ImagerSetup& s, int image_size, int correction, const GridOut& g, void* d_image,
    void* d_beam, int out_f32, ScalarPack* pack)
{
    using C = typename Cplx<R>::T;
    const int N = s.N;
    C* tw = c->buf<C>("fft_tw", tw_size(N));
    if (!c->memo("fft_tw", std::to_string(N) + "/" + std::to_string(sizeof(R)))) {
        int logm = 0;
        while ((2 << logm) < N)
            logm++;
        k_fft_tables<R><<<grid1d(tw_size(N), 256), 256, 0, c->stream>>>(N, logm, tw);
        STPGPU_CHECK_LAUNCH();
    }
    if (correction)
        device_gcf<R>(c, s);
    const double* ginv = correction ? c->buf<double>("gcfinv", N) : nullptr;
    auto one = [&](void* grid, void* out, ScalarPack* pk) {
        launch_axis<R, true>(c, g, grid, N, axis_n1(N), tw);
        launch_axis<R, false>(c, g, grid, N, N / axis_n1(N), tw);
        if (pk)
            c->mark(3);
        if constexpr (sizeof(R) == 8) {
            if (!out_f32) {
                launch_c2r<R, double>(c, s, image_size, correction, g, grid, tw, ginv, out, pk);
                return;
            }
        }
        launch_c2r<R, float>(c, s, image_size, correction, g, grid, tw, ginv, out, pk);
    };
    one(g.grid, d_image, pack);
    c->mark(4);
    if (s.beam && d_beam)
        one(g.beam, d_beam, nullptr);
}

// c2r FFT + crop/normalise of a gridded snapshot (fft.cpp:45-135,
// imager.h:97-213) on the context's current stream; the call's scalars go
// to `pack`.
template <typename R>
void finish_imager(stpgpu_context* c, const ImagerSetup& s, int image_size, int correction, const GridOut& g,
    void* d_image, void* d_beam, int out_f32, ScalarPack* pack)
{
    if constexpr (sizeof(R) == 4) {
        if (s.wide_fft) { // the gridder wrote double2 cells: Z2D + double normalisation
            finish_imager<double>(c, s, image_size, correction, g, d_image, d_beam, out_f32, pack);
            return;
        }
    }
    cudaStream_t st = c->stream;
    const int N = s.N;
    if (s.own_c2r) {
        finish_own<R>(c, s, image_size, correction, g, d_image, d_beam, out_f32, pack);
        return;
    }
    R* img = c->buf<R>("fftimg", size_t(N) * N);
    const cufftType type = sizeof(R) == 8 ? CUFFT_Z2D : CUFFT_C2R;
    cufftHandle h = c->plan(N, type);
    auto exec = [&](void* in, R* out) {
        cufftResult r;
        if (sizeof(R) == 8)
            r = cufftExecZ2D(h, reinterpret_cast<cufftDoubleComplex*>(in), reinterpret_cast<cufftDoubleReal*>(out));
        else
            r = cufftExecC2R(h, reinterpret_cast<cufftComplex*>(in), reinterpret_cast<cufftReal*>(out));
        if (r != CUFFT_SUCCESS)
            fail(STPGPU_ERR_CUFFT, "cuFFT c2r execution failed (" + std::to_string(int(r)) + ")");
    };
    const double* gcf = correction ? device_gcf<R>(c, s) : nullptr;
    const double* ginv = correction ? c->buf<double>("gcfinv", s.N) : nullptr;
    (void)gcf;
    const dim3 ngrid(std::min<unsigned>(grid1d(image_size, 256), 4), image_size);
    // 16-byte path: every 4-row group inside one crop segment and aligned
    const bool vec4 = (image_size % 8) == 0 && (N % 4) == 0
        && (reinterpret_cast<uintptr_t>(d_image) % 16) == 0 && (!d_beam || (reinterpret_cast<uintptr_t>(d_beam) % 16) == 0);
    const dim3 ngrid4(grid1d(image_size / 4, 256), (image_size + kNormCols - 1) / kNormCols);
    auto normalise = [&](void* out, ScalarPack* pk) {
        const PackArgs pa = pack_args(g, pk);
        if (vec4) {
            if (out_f32)
                k_normalise4<R, float><<<ngrid4, 256, 0, st>>>(img, N, image_size, g.d_total, ginv, correction,
                    reinterpret_cast<float*>(out), pa);
            else
                k_normalise4<R, double><<<ngrid4, 256, 0, st>>>(img, N, image_size, g.d_total, ginv, correction,
                    reinterpret_cast<double*>(out), pa);
            STPGPU_CHECK_LAUNCH();
            return;
        }
        if (out_f32)
            k_normalise<R, float><<<ngrid, 256, 0, st>>>(img, N, image_size, g.d_total, ginv, correction,
                reinterpret_cast<float*>(out), pa);
        else
            k_normalise<R, double><<<ngrid, 256, 0, st>>>(img, N, image_size, g.d_total, ginv, correction,
                reinterpret_cast<double*>(out), pa);
        STPGPU_CHECK_LAUNCH();
    };
    exec(g.grid, img);
    c->mark(3);
    normalise(d_image, pack);
    c->mark(4);
    if (s.beam && d_beam) {
        exec(g.beam, img);
        normalise(d_beam, nullptr);
    }
}

// Compensated FP32 keeps the grid in double and runs the c2r in double
// precision when the grid correction would amplify the single-precision
// transform's rounding past the 1e-5 peak-relative bound.  Normalisation
// divides pixel (i, j) by gcf[i] gcf[j] (imager.h:97-150), so an error that
// the FP32 c2r leaves at about 4e-10 of the peak (measured on an 8192^2
// PSWF image with analytic correction: 2.3e-5 of the peak at
// 1/gcf_min^2 = 6.2e4, against 2.2e-6 for an FP32 grid transformed in
// double) is multiplied by up to 1/gcf_min^2 over the output field.  Rule:
// wide when 1/gcf_min^2 > 4096, i.e. an expected FP32-c2r error above about
// 1.5e-6 of the peak.  GaussianSinc S=3 with the DFT correction (1/gcf_min^2
// = 890) keeps the FP32 transform; PSWF (1.5e4 with the DFT correction at
// S=3, 6.2e4 analytic) takes the wide one.  The gcf values are those of
// k_imgdom_kernel (ImgDomKernel, conv_func.h:351-412) over the kept field.
constexpr double kWideFftAmplification = 4096.0;

bool wide_fft_rule(const ImagerSetup& s, int image_size, int correction)
{
    if (!correction)
        return false;
    const int N = s.N, centre = N / 2, hs = image_size / 2;
    double gmin = 1e300;
    if (s.analytic) {
        for (int m = -hs; m < hs; m++)
            gmin = std::min(gmin, std::fabs(gcf_value(s.kf, double(m) / centre)));
    } else {
        const int dmax = int(std::floor(s.trunc)) + 1;
        const int dlo = -std::min(dmax, centre), dhi = std::min(dmax, N - centre - 1);
        double ssum = 0.0;
        for (int d = dlo; d <= dhi; d++)
            ssum += kernel_value(s.kf, s.trunc, double(d));
        const double kinv = ssum > 0.0 ? 1.0 / ssum : 1.0;
        for (int m = 0; m <= hs; m++) {
            double r = 0.0;
            for (int d = dlo; d <= dhi; d++) {
                const long long jm = (long long)(d < 0 ? d + N : d) * m % N;
                r += kernel_value(s.kf, s.trunc, double(d)) * kinv * std::cos(2.0 * M_PI * double(jm) / double(N));
            }
            gmin = std::min(gmin, std::fabs(r));
        }
    }
    return !(gmin > 0.0) || 1.0 / (gmin * gmin) > kWideFftAmplification;
}

// wide_fft_rule memoised for the process (the DFT form costs a few thousand
// cosines per evaluation); used by the imaging calls and the server's
// admission estimate
bool wide_fft_needed(const ImagerSetup& s, int image_size, int correction)
{
    static std::mutex mu;
    static std::map<std::string, bool> memo;
    const std::string key = std::to_string(s.kf) + "/" + fkey(s.trunc) + "/" + std::to_string(s.N) + "/"
        + std::to_string(s.analytic) + "/" + std::to_string(image_size) + "/" + std::to_string(correction);
    std::lock_guard<std::mutex> lock(mu);
    auto it = memo.find(key);
    if (it != memo.end())
        return it->second;
    const bool wide = wide_fft_rule(s, image_size, correction);
    memo[key] = wide;
    return wide;
}

// stp::image_visibilities (imager.h:233-376) on device buffers.  The whole
// pipeline is enqueued without a host round trip; the normalisation reads
// the sampling total on the device, and the scalars are read back once at
// the end (an empty result, imager.h:355, is reported then).
template <typename R, int COMP>
void run_imager(stpgpu_context* c, const ImagerSetup& s_in, int image_size, int correction, const void* d_vis,
    int vis_c64, const double* d_wts, const double* d_uvw, int64_t n, void* d_image, void* d_beam, int out_f32,
    stpgpu_imager_info* info, bool graphable = false)
{
    if (image_size <= 0 || image_size > s_in.N || (image_size % 2) != 0)
        fail(STPGPU_ERR_INVALID_ARG, "image_size must be even, > 0 and <= padded_image_size");
    ImagerSetup s = s_in;
    s.wide_fft = (COMP == 1 && wide_fft_needed(s, image_size, correction)) ? 1 : 0;
    s.own_c2r = own_c2r_applies(s, sizeof(R) == 8 || s.wide_fft, out_f32, d_image, d_beam);
    // W-planes without the |w| sort where they apply (mean |w| per plane, no
    // A-projection time steps); a size class whose data did not allow it on
    // its last call (visibilities outside the grid, non-finite w) sorts
    s.wsel = s.nplanes > 0 && s.nplanes <= WSEL_MAXP && !s.wmedian && s.ntimesteps == 0 && !s.full_wsort
        && n < (int64_t(1) << 31);
    const int precision = sizeof(R) == 8 ? STPGPU_FP64 : (COMP ? STPGPU_FP32C : STPGPU_FP32);
    const std::string cls = size_class(s, precision);
    if (s.wsel && c->wsel_off.count(cls))
        s.wsel = 0;
    GridOut g;
    ScalarPack* pack = c->host_stage_dev(c->host_stage<ScalarPack>(1));
    // Device-pointer calls that repeat the previous call exactly (parameters,
    // sizes, buffers) replay a CUDA graph of the gridding, FFT and
    // normalisation kernels, captured on the first repeat; any other call
    // drops it.  The data in the buffers may change between calls.
    std::string sig;
    if (graphable && !c->timing && !large_support(s) && s.ntimesteps == 0) {
        auto put = [&](const void* q, size_t nb) { sig.append(reinterpret_cast<const char*>(q), nb); };
        put(&precision, sizeof(precision));
        put(&s, sizeof(s));
        put(&image_size, sizeof(image_size));
        put(&correction, sizeof(correction));
        put(&vis_c64, sizeof(vis_c64));
        put(&n, sizeof(n));
        put(&out_f32, sizeof(out_f32));
        const void* ptrs[7] = { d_vis, d_wts, d_uvw, d_image, d_beam, pack, reinterpret_cast<const void*>(c->stream) };
        put(ptrs, sizeof(ptrs));
    }
    const bool repeat = !sig.empty() && sig == c->single_sig;
    if (!repeat)
        c->drop_single();
    if (repeat && c->single_exec) {
        STPGPU_CUDA_TRY(cudaGraphLaunch(c->single_exec, c->stream));
        g_launches += c->single_launches; // the replay runs the captured kernels
        g = c->single_g;
    } else if (repeat) {
        const int before = g_launches;
        STPGPU_CUDA_TRY(cudaStreamBeginCapture(c->stream, cudaStreamCaptureModeThreadLocal));
        try {
            g = run_gridder<R, COMP>(c, s, d_vis, vis_c64, d_wts, d_uvw, 0, n);
            finish_imager<R>(c, s, image_size, correction, g, d_image, d_beam, out_f32, pack);
        } catch (...) {
            cudaGraph_t dead = nullptr;
            cudaStreamEndCapture(c->stream, &dead);
            if (dead)
                cudaGraphDestroy(dead);
            c->drop_single();
            throw;
        }
        STPGPU_CUDA_TRY(cudaStreamEndCapture(c->stream, &c->single_graph));
        int zk = 0;
        c->single_graph = memsets_to_kernels(c->single_graph, &zk);
        g_launches += zk;
        STPGPU_CUDA_TRY(cudaGraphInstantiate(&c->single_exec, c->single_graph, 0));
        STPGPU_CUDA_TRY(cudaGraphLaunch(c->single_exec, c->stream));
        c->single_g = g;
        c->single_launches = g_launches - before;
    } else {
        g = run_gridder<R, COMP>(c, s, d_vis, vis_c64, d_wts, d_uvw, 0, n);
    }
    if (!(repeat && c->single_exec))
        finish_imager<R>(c, s, image_size, correction, g, d_image, d_beam, out_f32, pack);
    if (!sig.empty())
        c->single_sig = sig;
    const int N = s.N;
    ScalarPack sb = read_back(c, g, true);
    if (sb.err & 16u) {
        // the W-planes without the sort did not apply: the sorting path, for
        // this call and the size class's next ones
        c->wsel_off.insert(cls);
        c->drop_single();
        s.wsel = 0;
        g = run_gridder<R, COMP>(c, s, d_vis, vis_c64, d_wts, d_uvw, 0, n);
        finish_imager<R>(c, s, image_size, correction, g, d_image, d_beam, out_f32, pack);
        sb = read_back(c, g, true);
    }
    if ((sb.err & 4u) && !s.full_wsort) {
        // rare data (many distinct |w| within one single-precision step): redo with the 64-bit |w| sort
        ImagerSetup s64 = s;
        s64.full_wsort = 1;
        g = run_gridder<R, COMP>(c, s64, d_vis, vis_c64, d_wts, d_uvw, 0, n);
        finish_imager<R>(c, s64, image_size, correction, g, d_image, d_beam, out_f32, pack);
        sb = read_back(c, g, true);
    }
    if (info) {
        info->sample_grid_total = sb.total;
        info->n_good_vis = int64_t(sb.ngood);
        info->n_grid_items = sb.nitems;
        info->padded_image_size = N;
        info->num_wplanes = s.nplanes;
        info->max_plane_support = sb.max_support;
        info->flags = s.wide_fft ? 1 : 0;
        info->image_size = sb.total > 0.0 ? image_size : 0;
        if (c->timing) {
            float ms[4] = { 0, 0, 0, 0 };
            for (int k = 0; k < 4; k++)
                STPGPU_CUDA_TRY(cudaEventElapsedTime(&ms[k], c->pev[k], c->pev[k + 1]));
            for (int k = 0; k < 4; k++)
                info->phase_ms[k] = ms[k];
        }
    }
}

ImagerSetup setup_from(const stpgpu_imager_pars* p, const stpgpu_wproj_pars* w, const stpgpu_aproj_pars* a,
    int& image_size)
{
    if (!p)
        fail(STPGPU_ERR_INVALID_ARG, "null imager parameters");
    if (p->kernel_function < 0 || p->kernel_function > 5)
        fail(STPGPU_ERR_INVALID_ARG, "unknown kernel function");
    if (!(p->cell_size > 0.0))
        fail(STPGPU_ERR_INVALID_ARG, "cell_size must be > 0");
    if (!(p->padding_factor >= 1.0))
        fail(STPGPU_ERR_INVALID_ARG, "padding_factor must be >= 1");
    ImagerSetup s;
    image_size = p->image_size;
    s.N = p->padded_image_size > 0 ? p->padded_image_size : int(unsigned(double(image_size) * p->padding_factor));
    s.kf = p->kernel_function;
    s.support = p->kernel_support;
    s.trunc = double(p->kernel_support);
    s.kernel_exact = p->kernel_exact;
    s.os = p->oversampling;
    s.beam = p->generate_beam;
    s.analytic = p->analytic_gcf;
    s.cell_size = p->cell_size;
    s.shift_uv = 1;
    s.halfplane = 1;
    if (w && w->num_wplanes > 0) {
        if (p->kernel_exact)
            fail(STPGPU_ERR_INVALID_ARG, "W-projection cannot be used with kernel_exact (imager.h:287)");
        s.nplanes = w->num_wplanes;
        s.max_support = w->max_wpconv_support;
        s.undersampling = w->undersampling_opt;
        s.trunc_perc = w->kernel_trunc_perc;
        s.wmedian = w->wplanes_median;
        if (w->hankel_opt) {
            // InterpType (types.h:55-59): LINEAR 0, CUBIC 1, COSINE 2 (interpolated linearly,
            // aw_projection.cpp:263-266)
            if (w->interp_type < 0 || w->interp_type > 2)
                fail(STPGPU_ERR_INVALID_ARG, "unknown interp_type");
            s.hankel = 1;
            s.proj_slice = w->hankel_proj_slice ? 1 : 0;
            s.cubic = w->interp_type == 1;
        }
    }
    if (!p->kernel_exact && p->oversampling < 1)
        fail(STPGPU_ERR_INVALID_ARG, "oversampling must be >= 1 when kernel_exact is false");
    if (a && a->num_timesteps > 0) {
        // imager.h:274-283
        if (s.nplanes <= 0)
            fail(STPGPU_ERR_INVALID_ARG, "W-projection must be used when A-projection is enabled.");
        if (s.hankel)
            fail(STPGPU_ERR_INVALID_ARG, "Hankel transform cannot be used when A-projection is enabled.");
        if (a->num_timesteps > 255 || int64_t(a->num_timesteps) * s.nplanes > 65535)
            fail(STPGPU_ERR_UNSUPPORTED, "A-projection supports at most 255 time steps and 65535 planes x steps");
        if (a->n_pbeam_coefs < 1 || !a->pbeam_coefs)
            fail(STPGPU_ERR_INVALID_ARG, "A-projection needs the primary beam coefficients");
        s.ntimesteps = a->num_timesteps;
        s.aproj_opt = a->aproj_opt ? 1 : 0;
        s.obs_dec = (a->obs_dec * M_PI) / 180.0; // deg2rad, global_macros.h:40
        s.obs_ra = (a->obs_ra * M_PI) / 180.0;
        s.lha = a->lha;
        s.pbcoefs = a->pbeam_coefs;
        s.npbcoefs = a->n_pbeam_coefs;
    }
    return s;
}

template <typename T>
T* to_device(stpgpu_context* c, const char* name, const void* host, size_t count)
{
    T* d = c->buf<T>(name, count);
    if (count)
        STPGPU_CUDA_TRY(cudaMemcpyAsync(d, host, sizeof(T) * count, cudaMemcpyHostToDevice, c->stream));
    return d;
}

// ------------------------------------------------------------------ batch

constexpr int kBatchStreams = 8;

struct BatchSnap {
    ImagerSetup s;
    int image_size = 0;
    int correction = 1;
    const void* vis = nullptr; // caller's pointers (device or host)
    int c64 = 0;
    const double* wts = nullptr;
    const double* uvw = nullptr;
    int64_t n = 0;
    void* image = nullptr;
    std::string cls; // size class
};

void batch_streams(stpgpu_context* c)
{
    if (!c->wstreams.empty())
        return;
    for (int k = 0; k < kBatchStreams; k++) {
        cudaStream_t w;
        STPGPU_CUDA_TRY(cudaStreamCreateWithFlags(&w, cudaStreamNonBlocking));
        c->wstreams.push_back(w);
        cudaEvent_t e;
        STPGPU_CUDA_TRY(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
        c->wevents.push_back(e);
    }
    STPGPU_CUDA_TRY(cudaEventCreateWithFlags(&c->fork_ev, cudaEventDisableTiming));
}

// main stream -> every worker stream
void batch_fork(stpgpu_context* c, cudaStream_t main)
{
    STPGPU_CUDA_TRY(cudaEventRecord(c->fork_ev, main));
    for (auto w : c->wstreams)
        STPGPU_CUDA_TRY(cudaStreamWaitEvent(w, c->fork_ev, 0));
}

// every worker stream -> main stream
void batch_join(stpgpu_context* c, cudaStream_t main)
{
    for (size_t k = 0; k < c->wstreams.size(); k++) {
        STPGPU_CUDA_TRY(cudaEventRecord(c->wevents[k], c->wstreams[k]));
        STPGPU_CUDA_TRY(cudaStreamWaitEvent(main, c->wevents[k], 0));
    }
}

// Enqueue one batch: every snapshot's whole pipeline (with host buffers, its
// transfers too) on its worker stream, so that the snapshots overlap, and the
// scalars of each written to `scal` (the device's address of pinned host
// memory).
template <typename R, int COMP>
void batch_enqueue(stpgpu_context* c, std::vector<BatchSnap>& B, int out_f32, int device_ptrs, ScalarPack* scal)
{
    const cudaStream_t main = c->stream;
    const int nb = int(B.size());
    const int K = int(c->wstreams.size());
    batch_fork(c, main);
    for (int i = 0; i < nb; i++) {
        c->stream = c->wstreams[i % K];
        c->ns = "b" + std::to_string(i) + "/";
        BatchSnap& b = B[i];
        const void* dv = b.vis;
        const double* dw = b.wts;
        const double* duvw = b.uvw;
        void* di = b.image;
        const size_t ob = (out_f32 ? 4 : 8) * size_t(b.image_size) * b.image_size;
        if (!device_ptrs) {
            dv = to_device<unsigned char>(c, "in_vis", b.vis, (b.c64 ? 8 : 16) * size_t(b.n));
            dw = to_device<double>(c, "in_w", b.wts, size_t(b.n));
            duvw = to_device<double>(c, "in_uvw", b.uvw, 3 * size_t(b.n));
            di = c->buf<unsigned char>("out_img", ob);
        }
        const GridOut g = run_gridder<R, COMP>(c, b.s, dv, b.c64, dw, duvw, 0, b.n);
        finish_imager<R>(c, b.s, b.image_size, b.correction, g, di, nullptr, out_f32, scal + i);
        if (!device_ptrs)
            STPGPU_CUDA_TRY(cudaMemcpyAsync(b.image, di, ob, cudaMemcpyDeviceToHost, c->stream));
    }
    c->stream = main;
    c->ns = "";
    batch_join(c, main);
}

template <typename R, int COMP>
void run_batch(stpgpu_context* c, const stpgpu_snapshot* sn, int nb, int precision, int out_f32, int device_ptrs,
    stpgpu_imager_info* infos, stpgpu_batch_info* bi)
{
    batch_streams(c);
    c->drop_single();
    std::vector<BatchSnap> B(nb);
    std::string sig;
    auto put = [&](const void* p, size_t n) { sig.append(reinterpret_cast<const char*>(p), n); };
    put(&precision, sizeof(int));
    put(&out_f32, sizeof(int));
    put(&device_ptrs, sizeof(int));
    for (int i = 0; i < nb; i++) {
        const stpgpu_snapshot& x = sn[i];
        BatchSnap& b = B[i];
        b.s = setup_from(&x.pars, &x.wproj, nullptr, b.image_size);
        if (x.pars.generate_beam)
            fail(STPGPU_ERR_UNSUPPORTED, "generate_beam is not supported by the batch path");
        if (b.image_size <= 0 || b.image_size > b.s.N || (b.image_size % 2) != 0)
            fail(STPGPU_ERR_INVALID_ARG, "snapshot " + std::to_string(i) + ": image_size must be even, > 0 and <= padded size");
        if (x.n_vis < 0 || (x.n_vis > 0 && (!x.vis || !x.weights || !x.uvw)) || !x.image)
            fail(STPGPU_ERR_INVALID_ARG, "snapshot " + std::to_string(i) + ": null buffer");
        if (x.vis_dtype != STPGPU_C128 && x.vis_dtype != STPGPU_C64)
            fail(STPGPU_ERR_INVALID_ARG, "snapshot " + std::to_string(i) + ": vis_dtype");
        b.correction = x.pars.gridding_correction;
        if (precision == STPGPU_FP32C)
            b.s.wide_fft = wide_fft_needed(b.s, b.image_size, b.correction) ? 1 : 0;
        // (host images go through an aligned device buffer)
        b.s.own_c2r = own_c2r_applies(b.s, precision == STPGPU_FP64 || b.s.wide_fft, out_f32,
            device_ptrs ? x.image : nullptr, nullptr);
        b.vis = x.vis;
        b.c64 = x.vis_dtype == STPGPU_C64;
        b.wts = x.weights;
        b.uvw = x.uvw;
        b.n = x.n_vis;
        b.image = x.image;
        b.cls = size_class(b.s, precision) + "/batch";
        // W-planes without the |w| sort where they apply (as in single calls)
        b.s.wsel = b.s.nplanes > 0 && b.s.nplanes <= WSEL_MAXP && !b.s.wmedian && b.s.ntimesteps == 0
            && x.n_vis < (int64_t(1) << 31) && !c->wsel_off.count(b.cls);
        put(&b.s.wsel, sizeof(b.s.wsel));
        put(&x.pars, sizeof(x.pars));
        put(&x.wproj, sizeof(x.wproj));
        put(&x.n_vis, sizeof(x.n_vis));
        put(&x.vis_dtype, sizeof(x.vis_dtype));
        put(&x.vis, sizeof(void*));
        put(&x.weights, sizeof(void*));
        put(&x.uvw, sizeof(void*));
        put(&x.image, sizeof(void*));
    }
    if (sig != c->batch_sig) {
        for (auto w : c->wstreams)
            STPGPU_CUDA_TRY(cudaStreamSynchronize(w));
        STPGPU_CUDA_TRY(cudaStreamSynchronize(c->stream));
        c->drop_graph();
        c->batch_sig = sig;
        c->batch_calls = 0;
    }
    c->batch_calls++;
    // pinned staging: the scalars read back
    const size_t need = pad256(sizeof(ScalarPack) * nb) + 4096;
    if (c->batch_host_cap < need) {
        if (c->batch_host) {
            for (auto w : c->wstreams)
                STPGPU_CUDA_TRY(cudaStreamSynchronize(w));
            STPGPU_CUDA_TRY(cudaStreamSynchronize(c->stream));
            c->drop_graph();
            cudaFreeHost(c->batch_host);
            c->batch_host = nullptr;
            c->batch_host_cap = 0;
        }
        STPGPU_CUDA_TRY(cudaMallocHost(&c->batch_host, need));
        c->batch_host_cap = need;
    }
    ScalarPack* scal = reinterpret_cast<ScalarPack*>(c->batch_host);
    ScalarPack* scal_dev = nullptr;
    STPGPU_CUDA_TRY(cudaHostGetDevicePointer(reinterpret_cast<void**>(&scal_dev), scal, 0));
    const bool saved_timing = c->timing;
    c->timing = false;
    struct Restore {
        stpgpu_context* c;
        cudaStream_t main;
        bool timing;
        ~Restore()
        {
            c->stream = main;
            c->ns = "";
            c->timing = timing;
        }
    } restore { c, c->stream, saved_timing };
    const cudaStream_t main = c->stream;
    int graph = 0;
    g_launches = 0;
    if (device_ptrs && c->batch_exec) {
        // replay
        STPGPU_CUDA_TRY(cudaEventRecord(c->ev0, main));
        STPGPU_CUDA_TRY(cudaGraphLaunch(c->batch_exec, main));
        STPGPU_CUDA_TRY(cudaEventRecord(c->ev1, main));
        g_launches = c->batch_launches; // the replay runs the captured kernels
        graph = 1;
    } else {
        bool capturable = true;
        for (auto& b : B)
            capturable = capturable && !large_support(b.s);
        if (device_ptrs && capturable && c->batch_calls >= 2) {
            // capture the batch (buffers, plans and tables exist from the previous call)
            STPGPU_CUDA_TRY(cudaStreamBeginCapture(main, cudaStreamCaptureModeThreadLocal));
            try {
                batch_enqueue<R, COMP>(c, B, out_f32, device_ptrs, scal_dev);
            } catch (...) {
                cudaGraph_t g = nullptr;
                cudaStreamEndCapture(main, &g);
                if (g)
                    cudaGraphDestroy(g);
                throw;
            }
            STPGPU_CUDA_TRY(cudaStreamEndCapture(main, &c->batch_graph));
            int zk = 0;
            c->batch_graph = memsets_to_kernels(c->batch_graph, &zk);
            g_launches += zk;
            c->batch_launches = g_launches;
            STPGPU_CUDA_TRY(cudaGraphInstantiate(&c->batch_exec, c->batch_graph, 0));
            STPGPU_CUDA_TRY(cudaEventRecord(c->ev0, main));
            STPGPU_CUDA_TRY(cudaGraphLaunch(c->batch_exec, main));
            STPGPU_CUDA_TRY(cudaEventRecord(c->ev1, main));
            graph = 1;
        } else {
            STPGPU_CUDA_TRY(cudaEventRecord(c->ev0, main));
            batch_enqueue<R, COMP>(c, B, out_f32, device_ptrs, scal_dev);
            STPGPU_CUDA_TRY(cudaEventRecord(c->ev1, main));
        }
    }
    STPGPU_CUDA_TRY(cudaStreamSynchronize(main));
    for (int round = 0; round < 2; round++) {
        bool redo = false;
        for (int i = 0; i < nb; i++) {
            if (scal[i].err & 16u) { // the W-planes without the sort did not apply: the sorting path
                B[i].s.wsel = 0;
                c->wsel_off.insert(B[i].cls);
                redo = true;
            } else if (scal[i].err & 4u) { // long run of distinct |w| in the 24-bit sort: the 64-bit sort
                B[i].s.full_wsort = 1;
                redo = true;
            }
        }
        if (!redo)
            break;
        c->drop_graph();
        c->batch_calls = 0;
        c->batch_sig.clear();
        STPGPU_CUDA_TRY(cudaEventRecord(c->ev0, main));
        batch_enqueue<R, COMP>(c, B, out_f32, device_ptrs, scal_dev);
        STPGPU_CUDA_TRY(cudaEventRecord(c->ev1, main));
        STPGPU_CUDA_TRY(cudaStreamSynchronize(main));
        graph = 0;
    }
    float ms = 0.f;
    STPGPU_CUDA_TRY(cudaEventElapsedTime(&ms, c->ev0, c->ev1));
    for (int i = 0; i < nb; i++) {
        if (scal[i].err & ~4u)
            fail(STPGPU_ERR_DEVICE, "snapshot " + std::to_string(i) + ": gridder reported internal error flags "
                    + std::to_string(scal[i].err));
        if (infos) {
            stpgpu_imager_info& f = infos[i];
            std::memset(&f, 0, sizeof(f));
            f.sample_grid_total = scal[i].total;
            f.n_good_vis = int64_t(scal[i].ngood);
            f.n_grid_items = scal[i].nitems;
            f.padded_image_size = B[i].s.N;
            f.num_wplanes = B[i].s.nplanes;
            f.max_plane_support = scal[i].max_support;
            f.image_size = scal[i].total > 0.0 ? B[i].image_size : 0;
            f.flags = B[i].s.wide_fft ? 1 : 0;
        }
    }
    if (bi) {
        std::memset(bi, 0, sizeof(*bi));
        bi->device_ms = ms;
        bi->graph = graph;
        bi->gridder_launches = nb;
        bi->tuned_classes = 0;
        bi->n_launches = g_launches;
    }
}

// ------------------------------------------------------------------ source finder

// Exact k-th order statistic (0-based) by 16-bit radix select.
template <typename T>
double select_kth(stpgpu_context* c, const T* x, int64_t n, unsigned long long k)
{
    cudaStream_t st = c->stream;
    unsigned int* hist = c->buf<unsigned int>("rsel_hist", 65536);
    unsigned long long* state = c->buf<unsigned long long>("rsel_state", 3);
    unsigned long long h0[3] = { k, 0ull, 0ull };
    STPGPU_CUDA_TRY(cudaMemcpyAsync(state, h0, sizeof(h0), cudaMemcpyHostToDevice, st));
    unsigned long long* hs = c->host_stage<unsigned long long>(3);
    for (int pass = 3; pass >= 0; pass--) {
        const int shift = pass * 16;
        STPGPU_CUDA_TRY(cudaMemsetAsync(hist, 0, sizeof(unsigned int) * 65536, st));
        // prefix/mask are read on the host after each pass
        STPGPU_CUDA_TRY(cudaMemcpyAsync(hs, state, sizeof(h0), cudaMemcpyDeviceToHost, st));
        STPGPU_CUDA_TRY(cudaStreamSynchronize(st));
        k_radix_hist<T><<<std::min<unsigned>(grid1d(n, SF_THREADS), 148 * 16), SF_THREADS, 0, st>>>(x, n, hs[1],
            hs[2], shift, hist);
        STPGPU_CHECK_LAUNCH();
        k_radix_pick<<<1, 1024, 0, st>>>(hist, shift, state);
        STPGPU_CHECK_LAUNCH();
    }
    STPGPU_CUDA_TRY(cudaMemcpyAsync(hs, state, sizeof(h0), cudaMemcpyDeviceToHost, st));
    STPGPU_CUDA_TRY(cudaStreamSynchronize(st));
    // key -> double
    const unsigned long long key = hs[1];
    const unsigned long long u = (key >> 63) ? (key & 0x7fffffffffffffffull) : ~key;
    double v;
    std::memcpy(&v, &u, sizeof(v));
    return v;
}

// mat_median_exact (matrix_math.cpp:20-48)
template <typename T>
double median_exact(stpgpu_context* c, const T* x, int64_t n)
{
    const unsigned long long k = (unsigned long long)(n / 2);
    const double v1 = select_kth(c, x, n, k);
    if (n & 1)
        return v1;
    const double v2 = select_kth(c, x, n, k - 1);
    return (v1 + v2) / 2;
}

// Gaussian2dParams::convert_to_constrained_parameters (fitting.cpp:32-57)
void constrain(double* g)
{
    const double half_pi = M_PI / 2.0;
    g[3] = std::fabs(g[3]);
    g[4] = std::fabs(g[4]);
    if (g[3] < g[4]) {
        std::swap(g[3], g[4]);
        g[5] += half_pi;
    }
    double t = std::fmod(g[5], M_PI);
    if (t <= -half_pi)
        t += M_PI;
    else if (t > half_pi)
        t -= M_PI;
    g[5] = t;
}

// IslandParams::estimate_moments_fit (sourcefind.cpp:691-717)
void moments_fit(int sign, double extremum, const double* mb, double rms, double ana_sigma, double* g)
{
    const double xx = mb[2], yy = mb[3], xy = mb[4];
    const double w1 = (xx + yy) / 2.0;
    const double w2 = std::sqrt(((xx - yy) * (xx - yy) / 4) + xy * xy);
    const double tmaj = w1 + w2, tmin = w1 - w2;
    const double thr = ana_sigma * rms;
    const double ratio = sign * extremum / thr;
    const double scale = 1.0 - std::log(ratio) / (ratio - 1.0);
    double theta = 0.5 * std::atan(2.0 * xy / (xx - yy));
    if (theta * xy < 0.0)
        theta += M_PI / 2.0;
    g[0] = extremum;
    g[1] = mb[0];
    g[2] = mb[1];
    g[3] = std::sqrt(tmaj / scale);
    g[4] = std::sqrt(tmin / scale);
    g[5] = theta;
    constrain(g);
}

// k_seg_sort_big uses SEG_BIG indices of dynamic shared memory (more than the
// default 48 KB): raise its limit once per device.
void set_seg_sort_smem()
{
    static std::atomic<uint64_t> done { 0 };
    int dev = 0;
    STPGPU_CUDA_TRY(cudaGetDevice(&dev));
    const uint64_t bit = uint64_t(1) << (dev & 63);
    if (done.load() & bit)
        return;
    STPGPU_CUDA_TRY(cudaFuncSetAttribute(k_seg_sort_big, cudaFuncAttributeMaxDynamicSharedMemorySize,
        int(SEG_BIG * sizeof(uint32_t))));
    done.fetch_or(bit);
}

// Device state of one source-finder call: labeller counters, pass tickets,
// statistics and the clipping state, cleared by one memset per call.
struct SfState {
    uint32_t misc[8]; // CclBufs::misc, then the valid-label count [4] and the island count [5]
    unsigned int tickets[4];
    uint32_t seg[3]; // label analysis: segment allocation cursor, labels with entries, labels for the one-block sort
    SfStats st;
    ClipState cs;
};

// Blocks of the fused statistics kernel for T on the context's device (the
// cooperative grid: one block per SM); 0 when it cannot be launched
// cooperatively.
template <typename T>
int sf_stats_grid(stpgpu_context* c)
{
    static std::mutex mu;
    static std::map<int, int> grid;
    std::lock_guard<std::mutex> lk(mu);
    auto it = grid.find(c->device);
    if (it != grid.end())
        return it->second;
    int coop = 0, sms = 0, per_sm = 0;
    STPGPU_CUDA_TRY(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, c->device));
    STPGPU_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, c->device));
    STPGPU_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_sf_stats<T>, SF_STATS_THREADS, 0));
    const int g = coop ? std::min(per_sm, 1) * sms : 0;
    grid[c->device] = g;
    return g;
}

// Images of at least this many samples take the fused statistics kernel;
// smaller ones the pass kernels.
constexpr int64_t kSfFusedMin = int64_t(1) << 16;

// The pass kernels for every image when STPGPU_SF_STATS=passes.
bool sf_passes_forced()
{
    const char* e = std::getenv("STPGPU_SF_STATS");
    return e && std::strcmp(e, "passes") == 0;
}

// The statistics' working buffers at the sizes enqueue_stats asks for, so
// that a call sizes them before it looks at its graph signature.
template <typename T>
void size_stats_buffers(stpgpu_context* c, int64_t n, const stpgpu_sf_pars& p)
{
    const bool est = !(std::fabs(p.rms_est) > 0.0);
    const int grid = sf_stats_grid<T>(c);
    if (grid > 0) {
        const int64_t G = int64_t(grid) * SF_STATS_THREADS;
        c->buf<double>("sf_part_fused", 8 * size_t(grid));
        if (est)
            c->buf<T>("sf_clip_lists", size_t(sf_band_cap(n, G)) * size_t(G));
    }
    const unsigned nb = std::min<unsigned>(grid1d(n, SF_THREADS), 148 * SF_STREAM_BLOCKS);
    c->buf<double>("sf_part", 3 * size_t(nb));
    c->buf<unsigned long long>("sf_bins", BINS_N + 2);
}

// Statistics and thresholds (sourcefind.cpp:280-301) enqueued into s->st;
// only the exact median (NTHELEMENT, BINMEDIAN, or exact = the binned
// median's fallback) waits on the host.  With `fused` (16-byte aligned
// images of at least kSfFusedMin samples) one cooperative launch of
// k_sf_stats does the passes; otherwise one kernel per pass.
template <typename T>
void enqueue_stats(stpgpu_context* c, const T* x, int64_t n, const stpgpu_sf_pars& p, SfState* s, bool exact,
    bool fused)
{
    cudaStream_t st = c->stream;
    const bool est = !(std::fabs(p.rms_est) > 0.0);
    const int grid = fused ? sf_stats_grid<T>(c) : 0;
    if (grid > 0 && n >= kSfFusedMin && (reinterpret_cast<uintptr_t>(x) & 15) == 0 && !sf_passes_forced()) {
        int do_sum = est, do_hist = 0;
        switch (p.median_method) {
        case STPGPU_ZEROMEDIAN:
            break;
        case STPGPU_BINAPPROX:
            if (!exact) {
                do_sum = 1;
                do_hist = 1;
                break;
            }
            [[fallthrough]];
        case STPGPU_BINMEDIAN:
            do_sum = 1;
            [[fallthrough]];
        case STPGPU_NTHELEMENT:
            k_sf_set_median<<<1, 1, 0, st>>>(&s->st, median_exact(c, x, n));
            STPGPU_CHECK_LAUNCH();
            break;
        default:
            fail(STPGPU_ERR_INVALID_ARG, "unknown median method");
        }
        const int64_t G = int64_t(grid) * SF_STATS_THREADS;
        int cap = est ? sf_band_cap(n, G) : 0;
        double* part = c->buf<double>("sf_part_fused", 8 * size_t(grid));
        unsigned long long* bins = c->buf<unsigned long long>("sf_bins", BINS_N + 2);
        T* cand = est ? c->buf<T>("sf_clip_lists", size_t(cap) * size_t(G)) : nullptr;
        int iters = est ? p.sigma_clip_iters : 0;
        double rms = p.rms_est, ana = p.analysis_n_sigma, det = p.detection_n_sigma;
        const T* xa = x;
        SfStats* sta = &s->st;
        ClipState* csa = &s->cs;
        unsigned int* bar = &s->tickets[3];
        void* args[] = { (void*)&xa, (void*)&n, (void*)&sta, (void*)&csa, (void*)&part, (void*)&bins, (void*)&cand,
            (void*)&cap, (void*)&bar, (void*)&do_sum, (void*)&do_hist, (void*)&iters, (void*)&rms, (void*)&ana,
            (void*)&det };
        STPGPU_CUDA_TRY(cudaLaunchCooperativeKernel((const void*)k_sf_stats<T>, dim3(grid), dim3(SF_STATS_THREADS), args,
            0, st));
        return;
    }
    const unsigned nb = std::min<unsigned>(grid1d(n, SF_THREADS), 148 * SF_STREAM_BLOCKS);
    double* part = c->buf<double>("sf_part", 3 * size_t(nb));
    unsigned long long* bins = c->buf<unsigned long long>("sf_bins", BINS_N + 2);
    auto sum_sq = [&](bool with_bins) {
        k_sum_sq<T><<<nb, SF_THREADS, 0, st>>>(x, n, part, &s->tickets[0], &s->st, with_bins ? bins : nullptr);
        STPGPU_CHECK_LAUNCH();
    };
    auto set_median = [&](double m) {
        k_sf_set_median<<<1, 1, 0, st>>>(&s->st, m);
        STPGPU_CHECK_LAUNCH();
    };
    switch (p.median_method) {
    case STPGPU_ZEROMEDIAN: // the state starts at zero
        if (est)
            sum_sq(false);
        break;
    case STPGPU_BINAPPROX:
        if (!exact) {
            sum_sq(true);
            k_hist<T><<<nb, SF_THREADS, 0, st>>>(x, n, &s->st, bins, &s->tickets[1]);
            STPGPU_CHECK_LAUNCH();
            break;
        }
        [[fallthrough]];
    case STPGPU_BINMEDIAN: // successive binning ends in nth_element: the exact median
        sum_sq(false);
        set_median(median_exact(c, x, n));
        break;
    case STPGPU_NTHELEMENT:
        set_median(median_exact(c, x, n));
        if (est)
            sum_sq(false);
        break;
    default:
        fail(STPGPU_ERR_INVALID_ARG, "unknown median method");
    }
    if (est) {
        k_clip_init<<<1, 1, 0, st>>>(&s->cs, &s->st, double(n), 3.0);
        STPGPU_CHECK_LAUNCH();
        for (int it = 0; it < p.sigma_clip_iters; it++) {
            k_clip_pass<T><<<nb, SF_THREADS, 0, st>>>(x, n, &s->st, &s->cs, part, &s->tickets[2], 3.0);
            STPGPU_CHECK_LAUNCH();
        }
    }
    k_sf_thresholds<<<1, 1, 0, st>>>(&s->st, est ? &s->cs : nullptr, p.rms_est, p.analysis_n_sigma,
        p.detection_n_sigma);
    STPGPU_CHECK_LAUNCH();
}

// Labeller buffers for n pixels in ccl_chunks(n) chunks.
struct CclBufs {
    uint8_t* cls; // ccl_chunks(n) * CCL_CHUNK bytes (background padding past n)
    uint32_t* P; // n union-find parents (foreground keys only)
    uint32_t* R; // n: label number of each root
    uint32_t* cnt; // 3 rows of ccl_chunks(n) + 1: positive roots, negative roots, foreground keys per chunk
    uint32_t* off; // their exclusive scans, same layout
    uint32_t* misc; // [0..2] the three totals, [3] union-find step-bound flag (zero before the call)
    uint32_t* fgl; // n: foreground keys in scan order, or null
    int32_t* L; // n: label map in memory order, or null
};

inline int64_t ccl_chunks(int64_t n) { return (n + CCL_CHUNK - 1) / CCL_CHUNK; }

// Enqueues the labeller (ccl.h:19-773 semantics, see the kernels) on st.
// Counts its launches; makes no allocation and throws nothing.
template <typename T>
cudaError_t ccl_enqueue(cudaStream_t st, const T* img, const CclGeom& g, const double* thr, double tp, double tn,
    int findneg, int conn4, int slice, const CclBufs& b)
{
    const int64_t n = int64_t(g.rows) * g.cols;
    const int64_t nch = ccl_chunks(n), npad = nch * CCL_CHUNK;
    const int stride = int(nch + 1);
    unsigned* err = b.misc + 3;
    if (g.rows % 4 == 0 && (reinterpret_cast<uintptr_t>(img) & 15) == 0) {
        const int64_t nu = npad / CCL_KPT;
        k_ccl_init16<T><<<unsigned(std::min<int64_t>(ceil_div(nu, SF_THREADS), 148 * 4)), SF_THREADS, 0, st>>>(img,
            g, thr, tp, tn, findneg, n / 4, nu, reinterpret_cast<uint4*>(b.cls), reinterpret_cast<uint4*>(b.P));
    } else {
        if (npad > n) {
            const cudaError_t e = cudaMemsetAsync(b.cls + n, 0, size_t(npad - n), st);
            if (e != cudaSuccess)
                return e;
        }
        k_ccl_init<T><<<grid1d(n, 256), 256, 0, st>>>(img, g, thr, tp, tn, findneg, b.cls, b.P);
    }
    k_ccl_union<<<unsigned(nch), SF_THREADS, 0, st>>>(b.cls, g, conn4, slice, b.P, err);
    k_ccl_flatten<<<unsigned(nch), SF_THREADS, 0, st>>>(b.cls, b.P, b.cnt, stride, err);
    k_scan_rows<<<3, 1024, 0, st>>>(b.cnt, b.off, int(nch), stride, b.misc);
    k_ccl_rank<<<unsigned(nch), SF_THREADS, 0, st>>>(b.cls, b.P, b.off, stride, b.R, b.fgl);
    g_launches += 5;
    if (b.L) {
        if (g.rows % 4 == 0 && (reinterpret_cast<uintptr_t>(b.L) & 15) == 0) {
            const int64_t ng = n / 4;
            k_ccl_label16<<<unsigned(std::min<int64_t>(ceil_div(ceil_div(ng, 4), SF_THREADS), 148 * 8)), SF_THREADS,
                0, st>>>(b.cls, b.P, b.R, g, ng, b.L);
        } else {
            k_ccl_label<<<grid1d(n, 256), 256, 0, st>>>(b.cls, b.P, b.R, g, b.L);
        }
        g_launches++;
    }
    return cudaGetLastError();
}

// write_labels: fill the label map (d_labels, or the context's "ccl_L"
// buffer when d_labels is null).
template <typename T>
void run_source_find(stpgpu_context* c, const T* d_img, int rows, int cols, const stpgpu_sf_pars& p, int32_t* d_labels,
    bool write_labels, std::vector<stpgpu_island>& islands, stpgpu_sf_info& info)
{
    if (rows <= 0 || cols <= 0 || (rows % 2) || (cols % 2))
        fail(STPGPU_ERR_INVALID_ARG, "image dimensions must be positive and even (ccl.h:116-117)");
    if (rows > 65536 || cols > 65536 || int64_t(rows) * cols >= (int64_t(1) << 32))
        fail(STPGPU_ERR_INVALID_ARG, "image too large for the labeler (ccl.h:118-119)");
    cudaStream_t st = c->stream;
    const int64_t n = int64_t(rows) * cols;
    // ---- connected components
    const CclGeom geom { rows, cols, rows / 2, cols / 2 };
    const int64_t nch = ccl_chunks(n);
    CclBufs cb;
    cb.cls = c->buf<uint8_t>("ccl_cls", size_t(nch) * CCL_CHUNK);
    cb.P = c->buf<uint32_t>("ccl_P", n);
    cb.R = c->buf<uint32_t>("ccl_R", n);
    cb.cnt = c->buf<uint32_t>("ccl_cnt", 3 * size_t(nch + 1));
    cb.off = c->buf<uint32_t>("ccl_off", 3 * size_t(nch + 1));
    cb.fgl = c->buf<uint32_t>("ccl_fgl", n);
    cb.L = write_labels ? (d_labels ? d_labels : c->buf<int32_t>("ccl_L", n)) : nullptr;
    SfState* sfs = c->buf<SfState>("sf_state", 1);
    cb.misc = sfs->misc;
    const int slice = p.ccl_slice_cols > 0 ? p.ccl_slice_cols : std::max(2, cols / 8);

    // ---- extrema, detection filter, moments (sourcefind.cpp:342-628) over
    // the foreground list, enqueued behind the labeller before its counts are
    // known: the buffers are sized by capacities (remembered per context),
    // and a call whose counts exceed them runs this stage again
    constexpr bool packed = sizeof(T) == 4;
    constexpr int kFirst = 512; // island records read back with the counts
    const unsigned G = 148 * 4; // grid of the label-analysis loops
    const uint32_t split_m = uint32_t(cols / 2) * uint32_t(rows);
    int32_t* zero_map = p.generate_labelmap ? cb.L : nullptr;
    uint32_t* nvalid = cb.misc + 4;
    uint32_t* nisl = cb.misc + 5;
    uint32_t* nvk = cb.misc + 6; // valid entries
    uint32_t* sort_overflow = cb.misc + 7;
    uint32_t lcap = uint32_t(std::min<int64_t>(n, std::max<int64_t>(c->sf_label_cap, std::max<int64_t>(65536, n / 64))));
    uint32_t fcap = uint32_t(std::min<int64_t>(n, std::max<int64_t>(c->sf_fg_cap, std::max<int64_t>(131072, n / 16))));
    unsigned long long *ext = nullptr, *eidx = nullptr, *vkeys = nullptr;
    double* mom = nullptr;
    int* ns = nullptr;
    uint32_t *sb = nullptr, *se = nullptr, *sp = nullptr, *fcode = nullptr, *fm = nullptr, *v1 = nullptr;
    uint32_t *cursor = nullptr, *slots = nullptr, *bigl = nullptr, *listed = nullptr;
    IslandRaw* raw = nullptr;
    auto size_buffers = [&] {
        // per label: extremum keys (single precision: value-and-index keys),
        // first indices, moments, sample counts, list segments; per list
        // entry: label code, memory index, valid keys, sorted memory indices
        ext = c->buf<unsigned long long>("sf_ext", lcap);
        eidx = c->buf<unsigned long long>("sf_eidx", lcap);
        mom = c->buf<double>("sf_mom", 6 * size_t(lcap));
        ns = c->buf<int>("sf_ns", lcap);
        sb = c->buf<uint32_t>("fg_sb", lcap);
        se = c->buf<uint32_t>("fg_se", lcap);
        sp = c->buf<uint32_t>("fg_sp", lcap);
        raw = c->buf<IslandRaw>("sf_raw", std::max<uint32_t>(lcap, kFirst));
        fcode = c->buf<uint32_t>("fg_code", fcap);
        fm = c->buf<uint32_t>("fg_m", fcap);
        vkeys = c->buf<unsigned long long>("fg_vkeys", fcap);
        v1 = c->buf<uint32_t>("fg_v1", fcap);
        cursor = c->buf<uint32_t>("fg_cur", lcap);
        slots = c->buf<uint32_t>("fg_slots", fcap);
        bigl = c->buf<uint32_t>("fg_big", lcap);
        listed = c->buf<uint32_t>("fg_listed", lcap);
    };
    auto moments_and_islands = [&](const FgSizes& z, uint32_t longest) {
        k_label_sums<T><<<G, 32 * kSumWarps, 0, st>>>(z, d_img, rows, cols, v1, sb, se, sp, listed, &sfs->seg[1], longest,
            mom, ns);
        STPGPU_CHECK_LAUNCH();
        k_islands<packed><<<G, 256, 0, st>>>(z, &sfs->st, ext, eidx, ns, mom, p.source_min_area, nvalid, nisl, raw);
        STPGPU_CHECK_LAUNCH();
    };
    auto enqueue_analysis = [&] {
        const FgSizes z { cb.misc, lcap, fcap };
        k_fg_init<packed><<<G, 256, 0, st>>>(z, &sfs->st, ext, packed ? nullptr : eidx, sb, se, sp);
        STPGPU_CHECK_LAUNCH();
        k_fg_gather<T, packed><<<G, 256, 0, st>>>(z, d_img, cb.cls, cb.P, cb.R, geom, cb.fgl, fcode, fm, ext);
        STPGPU_CHECK_LAUNCH();
        if constexpr (!packed) {
            k_fg_extrema_idx<T><<<G, 256, 0, st>>>(z, &sfs->st, d_img, fcode, fm, ext, eidx);
            STPGPU_CHECK_LAUNCH();
        }
        k_fg_keys<packed><<<G, 256, 0, st>>>(z, &sfs->st, fcode, fm, ext, vkeys, nvk, zero_map, se);
        STPGPU_CHECK_LAUNCH();
        // ordered (deterministic) moments: each valid label's entries in a
        // range of their own, ordered by list position (one warp per label,
        // one block for the large ones), per-label sums in memory order;
        // island records appended in any order
        k_seg_alloc<<<G, 256, 0, st>>>(z, sb, se, cursor, &sfs->seg[0], listed);
        STPGPU_CHECK_LAUNCH();
        k_seg_scatter<<<G, 256, 0, st>>>(vkeys, nvk, cursor, slots);
        STPGPU_CHECK_LAUNCH();
        k_seg_sort<<<G, 256, 0, st>>>(listed, &sfs->seg[1], sb, se, slots, fm, split_m, v1, sp, bigl, &sfs->seg[2]);
        STPGPU_CHECK_LAUNCH();
        set_seg_sort_smem();
        k_seg_sort_big<<<64, 1024, SEG_BIG * sizeof(uint32_t), st>>>(sb, se, slots, fm, split_m, v1, sp, bigl,
            &sfs->seg[2], sort_overflow);
        STPGPU_CHECK_LAUNCH();
        moments_and_islands(z, SEG_BIG);
    };
    // everything, then one read-back: state (statistics, counts, flags) and
    // the first island records
    unsigned char* hb = c->host_stage<unsigned char>(sizeof(SfState) + 64 + sizeof(IslandRaw) * size_t(kFirst));
    SfState* hstate = reinterpret_cast<SfState*>(hb);
    IslandRaw* hfirst = reinterpret_cast<IslandRaw*>(hb + ((sizeof(SfState) + 63) / 64) * 64);
    // the state and the first island records (as many as the call found, up
    // to kFirst) written by one kernel straight into the page-locked stage
    static_assert(sizeof(SfState) % 4 == 0 && (sizeof(IslandRaw) * kFirst) % 16 == 0, "copy-out units");
    auto enqueue_copy_out = [&] {
        k_copy_out<<<unsigned((sizeof(IslandRaw) * kFirst / 16 + 255) / 256), 256, 0, st>>>(
            reinterpret_cast<const uint32_t*>(sfs), c->host_stage_dev(reinterpret_cast<uint32_t*>(hstate)),
            int(sizeof(SfState) / 4), reinterpret_cast<const uint4*>(raw),
            c->host_stage_dev(reinterpret_cast<uint4*>(hfirst)), int(sizeof(IslandRaw) * kFirst / 16),
            int(offsetof(SfState, misc) / 4) + 5, int(sizeof(IslandRaw)));
        STPGPU_CHECK_LAUNCH();
    };
    auto read_back_state = [&] {
        enqueue_copy_out();
        STPGPU_CUDA_TRY(cudaStreamSynchronize(st));
    };
    size_buffers();
    auto enqueue_attempt = [&](bool exact_median, bool fused_stats) {
        static_assert(sizeof(SfState) % 4 == 0, "SfState in 32-bit words");
        zero_words(st, { { sfs, int64_t(sizeof(SfState) / 4) } });
        enqueue_stats<T>(c, d_img, n, p, sfs, exact_median, fused_stats);
        STPGPU_CUDA_TRY(ccl_enqueue<T>(st, d_img, geom, sfs->st.thr, 0.0, 0.0, p.find_negative_sources,
            p.ccl_4connectivity, slice, cb));
        enqueue_analysis();
        enqueue_copy_out();
    };
    // The first attempt of a call identical to the previous one (same
    // buffers, sizes, parameters and capacities, no reallocation since)
    // replays a CUDA graph of it; the second such call captures it.  Calls
    // whose median needs the host (NTHELEMENT, BINMEDIAN) run eagerly, as does
    // every call after a capture that the runtime refused.
    size_stats_buffers<T>(c, n, p);
    std::string sig;
    if (!c->timing && !c->sf_graph_off
        && (p.median_method == STPGPU_ZEROMEDIAN || p.median_method == STPGPU_BINAPPROX)) {
        auto put = [&](const void* q, size_t nb) { sig.append(reinterpret_cast<const char*>(q), nb); };
        const int tsize = int(sizeof(T));
        const int forced = sf_passes_forced() ? 1 : 0;
        const int wl = write_labels ? 1 : 0;
        put(&tsize, sizeof(tsize));
        put(&rows, sizeof(rows));
        put(&cols, sizeof(cols));
        put(&p, sizeof(p));
        put(&wl, sizeof(wl));
        put(&forced, sizeof(forced));
        put(&lcap, sizeof(lcap));
        put(&fcap, sizeof(fcap));
        put(&c->buf_gen, sizeof(c->buf_gen));
        const void* ptrs[4] = { d_img, d_labels, hb, reinterpret_cast<const void*>(st) };
        put(ptrs, sizeof(ptrs));
    }
    const bool repeat = !sig.empty() && sig == c->sf_sig;
    if (!repeat) {
        c->drop_sf_graph();
        c->sf_sig = sig;
    }
    bool exact = false, fused = true;
    for (int attempt = 0; attempt < 3; attempt++) {
        // again when the binned median does not apply (the exact median), or
        // when the fused statistics kernel gave up at a barrier (the pass
        // kernels)
        if (attempt == 0 && repeat && c->sf_exec) {
            STPGPU_CUDA_TRY(cudaGraphLaunch(c->sf_exec, st));
            g_launches += c->sf_launches;
        } else if (attempt == 0 && repeat) {
            const int before = g_launches;
            bool captured = false;
            STPGPU_CUDA_TRY(cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal));
            try {
                enqueue_attempt(false, true);
                STPGPU_CUDA_TRY(cudaStreamEndCapture(st, &c->sf_graph));
                STPGPU_CUDA_TRY(cudaGraphInstantiate(&c->sf_exec, c->sf_graph, 0));
                captured = true;
            } catch (const Error&) {
                cudaGraph_t dead = nullptr;
                cudaStreamEndCapture(st, &dead); // ends a capture still open; fails harmlessly otherwise
                if (dead)
                    cudaGraphDestroy(dead);
                (void)cudaGetLastError();
                c->drop_sf_graph();
                c->sf_graph_off = true;
            }
            if (captured) {
                c->sf_launches = g_launches - before;
                STPGPU_CUDA_TRY(cudaGraphLaunch(c->sf_exec, st));
            } else {
                g_launches = before;
                enqueue_attempt(false, true);
            }
        } else {
            enqueue_attempt(exact, fused);
        }
        STPGPU_CUDA_TRY(cudaStreamSynchronize(st));
        if (hstate->st.stats_err && fused) {
            fused = false;
            continue;
        }
        if (hstate->st.need_exact && !exact) {
            exact = true;
            continue;
        }
        break;
    }
    if (hstate->st.stats_err)
        fail(STPGPU_ERR_DEVICE, "source-finder statistics failed");
    if (hstate->misc[3])
        fail(STPGPU_ERR_DEVICE, "labeler gave up (union-find step bound)");
    const int np = int(hstate->misc[0]), nneg = int(hstate->misc[1]), nfg = int(hstate->misc[2]);
    const int nl = std::max(1, np + nneg);
    if (uint32_t(np + nneg) > lcap || uint32_t(nfg) > fcap) {
        // counts beyond the capacities: larger buffers, the stage again
        lcap = uint32_t(std::max<int64_t>(lcap, np + nneg + (np + nneg) / 4));
        fcap = uint32_t(std::max<int64_t>(fcap, nfg + nfg / 4));
        lcap = uint32_t(std::min<int64_t>(lcap, n));
        fcap = uint32_t(std::min<int64_t>(fcap, n));
        size_buffers();
        STPGPU_CUDA_TRY(cudaMemsetAsync(cb.misc + 4, 0, 4 * sizeof(uint32_t), st));
        STPGPU_CUDA_TRY(cudaMemsetAsync(sfs->seg, 0, sizeof(sfs->seg), st));
        enqueue_analysis();
        read_back_state();
    }
    c->sf_label_cap = std::max<uint32_t>(c->sf_label_cap, lcap);
    c->sf_fg_cap = std::max<uint32_t>(c->sf_fg_cap, fcap);
    if (hstate->misc[7]) {
        // a label with more valid entries than the one-block sort holds:
        // sort all entries with the multi-block sort, then sums and islands
        // again
        const uint32_t nv = hstate->misc[6];
        int end_bit = 33;
        while (end_bit < 64 && (uint64_t(1) << (end_bit - 32)) <= uint64_t(nl))
            end_bit++;
        unsigned long long* vk2 = c->buf<unsigned long long>("fg_vkeys2", nv);
        size_t tb = 0;
        cub::DeviceRadixSort::SortKeys(nullptr, tb, vkeys, vk2, int(nv), 0, end_bit, st);
        void* tmp = c->buf<unsigned char>("cubtmp_sf", tb);
        if (cub::DeviceRadixSort::SortKeys(tmp, tb, vkeys, vk2, int(nv), 0, end_bit, st) != cudaSuccess)
            fail(STPGPU_ERR_CUDA, "label sort failed");
        k_seg_mark<<<grid1d(nv, 256), 256, 0, st>>>(vk2, nv, fm, split_m, v1, sb, se, sp);
        STPGPU_CHECK_LAUNCH();
        STPGPU_CUDA_TRY(cudaMemsetAsync(cb.misc + 4, 0, 2 * sizeof(uint32_t), st));
        moments_and_islands(FgSizes { cb.misc, lcap, fcap }, ~0u);
        read_back_state();
    }
    const SfState h = *hstate;
    info.bg_level = h.st.median;
    info.rms_est = h.st.rms;
    info.mean = h.st.mean;
    info.sigma = h.st.sigma;
    const double rms = h.st.rms;
    info.n_labels_pos = np;
    info.n_labels_neg = nneg;
    const int first = std::min(nl, kFirst);
    const uint32_t* fit_pix = h.misc[6] > 0 ? v1 : nullptr;
    const int nis = int(h.misc[5]);
    info.n_valid_labels = int(h.misc[4]);
    info.n_islands = nis;
    std::vector<IslandRaw> hr(nis);
    std::copy(hfirst, hfirst + std::min(nis, first), hr.begin());
    if (nis > first) {
        STPGPU_CUDA_TRY(cudaMemcpyAsync(hr.data() + first, raw + first, sizeof(IslandRaw) * (nis - first),
            cudaMemcpyDeviceToHost, st));
        STPGPU_CUDA_TRY(cudaStreamSynchronize(st));
    }
    // label order: positives by label, then negatives
    std::sort(hr.begin(), hr.end(), [](const IslandRaw& a, const IslandRaw& b) {
        const bool na = a.label < 0, nb = b.label < 0;
        if (na != nb)
            return nb;
        return std::abs(a.label) < std::abs(b.label);
    });
    islands.resize(nis);
    const int vs = rows / 2, hs = cols / 2;
    for (int i = 0; i < nis; i++) {
        const IslandRaw& r = hr[i];
        stpgpu_island& o = islands[i];
        std::memset(&o, 0, sizeof(o));
        o.label_idx = r.label;
        o.sign = r.label < 0 ? -1 : 1;
        o.extremum_val = r.extremum_val;
        const int row = int(r.extremum_idx % rows), col = int(r.extremum_idx / rows);
        o.extremum_y_idx = row < vs ? row + vs : row - vs; // sourcefind.cpp:243-244
        o.extremum_x_idx = col < hs ? col + hs : col - hs;
        o.num_samples = r.num_samples;
        // moment normalisation (sourcefind.cpp:591-604)
        const double* a = r.mom;
        double mb[5];
        mb[0] = a[0] / a[5];
        mb[1] = a[1] / a[5];
        mb[2] = a[2] / a[5] - mb[0] * mb[0];
        mb[3] = a[3] / a[5] - mb[1] * mb[1];
        mb[4] = a[4] / a[5] - mb[0] * mb[1];
        moments_fit(o.sign, o.extremum_val, mb, rms, p.analysis_n_sigma, o.moments_fit);
    }
    if (p.gaussian_fitting && nis > 0) {
        // least-squares 2-D Gaussian per island (sourcefind.cpp:719-866): islands of one or two pixels keep
        // (extremum, 0, ...); the others start from the moments fit, unset widths as 1
        std::vector<int> keys, which;
        std::vector<double> init;
        for (int i = 0; i < nis; i++) {
            stpgpu_island& o = islands[i];
            if (o.num_samples < 3) {
                o.leastsq_fit[0] = o.extremum_val;
                continue;
            }
            const int l = o.label_idx;
            keys.push_back(l > 0 ? l - 1 : np + (-l - 1));
            which.push_back(i);
            const double* m = o.moments_fit;
            const double g[6] = { m[0], m[1], m[2], m[3] > 0.0 ? m[3] : 1.0, m[4] > 0.0 ? m[4] : 1.0, m[5] };
            init.insert(init.end(), g, g + 6);
        }
        const int nfit = int(keys.size());
        if (nfit > 0 && fit_pix) {
            int* dkeys = c->buf<int>("fit_keys", nfit);
            double* dinit = c->buf<double>("fit_init", 6 * size_t(nfit));
            double* dout = c->buf<double>("fit_out", 6 * size_t(nfit));
            int* dit = c->buf<int>("fit_iter", nfit);
            STPGPU_CUDA_TRY(cudaMemcpyAsync(dkeys, keys.data(), sizeof(int) * nfit, cudaMemcpyHostToDevice, st));
            STPGPU_CUDA_TRY(cudaMemcpyAsync(dinit, init.data(), sizeof(double) * 6 * nfit, cudaMemcpyHostToDevice, st));
            k_gauss_fit<T><<<nfit, FIT_THREADS, 0, st>>>(d_img, rows, cols, fit_pix, sb, se, sp, dkeys, dinit, nfit, dout, dit);
            STPGPU_CHECK_LAUNCH();
            std::vector<double> out(6 * size_t(nfit));
            std::vector<int> its(nfit);
            STPGPU_CUDA_TRY(cudaMemcpyAsync(out.data(), dout, sizeof(double) * 6 * nfit, cudaMemcpyDeviceToHost, st));
            STPGPU_CUDA_TRY(cudaMemcpyAsync(its.data(), dit, sizeof(int) * nfit, cudaMemcpyDeviceToHost, st));
            STPGPU_CUDA_TRY(cudaStreamSynchronize(st));
            for (int k = 0; k < nfit; k++) {
                stpgpu_island& o = islands[which[k]];
                for (int q = 0; q < 6; q++)
                    o.leastsq_fit[q] = out[6 * size_t(k) + q];
                constrain(o.leastsq_fit); // fitting.cpp:32-57
                o.fit_iterations = its[k];
            }
        }
    }
}

} // namespace

// ====================================================================== C ABI

extern "C" {

int stpgpu_abi_version(void) { return STPGPU_ABI_VERSION; }

stpgpu_status stpgpu_create(int device, stpgpu_context** out)
{
    if (!out)
        return STPGPU_ERR_INVALID_ARG;
    *out = nullptr;
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev <= 0) {
        cudaGetLastError();
        return STPGPU_ERR_NO_DEVICE;
    }
    if (device < 0 || device >= ndev)
        return STPGPU_ERR_INVALID_ARG;
    stpgpu_context* c = new stpgpu_context();
    c->device = device;
    stpgpu_status s = guard(c, [&] {
        STPGPU_CUDA_TRY(cudaStreamCreateWithFlags(&c->stream, cudaStreamNonBlocking));
        STPGPU_CUDA_TRY(cudaEventCreate(&c->ev0));
        STPGPU_CUDA_TRY(cudaEventCreate(&c->ev1));
    });
    if (s != STPGPU_OK) {
        delete c;
        return s;
    }
    *out = c;
    return STPGPU_OK;
}

stpgpu_status stpgpu_destroy(stpgpu_context* c)
{
    if (!c)
        return STPGPU_OK;
    cudaSetDevice(c->device);
    c->release();
    if (c->pinned)
        cudaFreeHost(c->pinned);
    if (c->batch_host)
        cudaFreeHost(c->batch_host);
    for (auto w : c->wstreams)
        cudaStreamDestroy(w);
    for (auto e : c->wevents)
        cudaEventDestroy(e);
    if (c->fork_ev)
        cudaEventDestroy(c->fork_ev);
    if (c->ev0)
        cudaEventDestroy(c->ev0);
    if (c->ev1)
        cudaEventDestroy(c->ev1);
    for (auto& e : c->pev)
        if (e)
            cudaEventDestroy(e);
    if (c->stream)
        cudaStreamDestroy(c->stream);
    delete c;
    return STPGPU_OK;
}

const char* stpgpu_last_error(const stpgpu_context* c) { return c ? c->err.c_str() : "null context"; }

void* stpgpu_stream(stpgpu_context* c) { return c ? reinterpret_cast<void*>(c->stream) : nullptr; }

stpgpu_status stpgpu_trim(stpgpu_context* c)
{
    return guard(c, [&] { c->release(); });
}

stpgpu_status stpgpu_image_visibilities_ex(stpgpu_context* c, const void* vis, int vis_dtype, const double* weights,
    const double* uvw, int64_t n_vis, const stpgpu_imager_pars* pars, const stpgpu_wproj_pars* wproj,
    const stpgpu_aproj_pars* aproj, int precision, void* image, void* beam, int out_dtype, int device_ptrs,
    stpgpu_imager_info* info)
{
    return guard(c, [&] {
        int image_size = 0;
        ImagerSetup s = setup_from(pars, wproj, aproj, image_size);
        if (n_vis < 0 || (n_vis > 0 && (!vis || !weights || !uvw)) || !image)
            fail(STPGPU_ERR_INVALID_ARG, "null buffer");
        if (vis_dtype != STPGPU_C128 && vis_dtype != STPGPU_C64)
            fail(STPGPU_ERR_INVALID_ARG, "vis_dtype");
        if (out_dtype != STPGPU_F64 && out_dtype != STPGPU_F32)
            fail(STPGPU_ERR_INVALID_ARG, "out_dtype");
        const int vc64 = vis_dtype == STPGPU_C64;
        const size_t vbytes = vc64 ? 8 : 16;
        const void* dv = vis;
        const double* dw = weights;
        const double* duvw = uvw;
        const bool timed = !device_ptrs;
        if (timed)
            STPGPU_CUDA_TRY(cudaEventRecord(c->ev0, c->stream));
        if (s.ntimesteps > 0 && n_vis > 0 && !s.lha)
            fail(STPGPU_ERR_INVALID_ARG, "A-projection needs the hour angle of every visibility (lha)");
        if (!device_ptrs) {
            dv = to_device<unsigned char>(c, "in_vis", vis, vbytes * size_t(n_vis));
            dw = to_device<double>(c, "in_w", weights, size_t(n_vis));
            duvw = to_device<double>(c, "in_uvw", uvw, 3 * size_t(n_vis));
            if (s.ntimesteps > 0)
                s.lha = to_device<double>(c, "in_lha", s.lha, size_t(n_vis));
        }
        const int64_t npix = int64_t(image_size) * image_size;
        const size_t obytes = out_dtype == STPGPU_F32 ? 4 : 8;
        void* dimg = image;
        void* dbeam = beam;
        if (!device_ptrs) {
            dimg = c->buf<unsigned char>("out_img", obytes * size_t(std::max<int64_t>(npix, 1)));
            dbeam = (s.beam && beam) ? c->buf<unsigned char>("out_beam", obytes * size_t(std::max<int64_t>(npix, 1)))
                                     : nullptr;
        }
        stpgpu_imager_info local {};
        stpgpu_imager_info* inf = info ? info : &local;
        std::memset(inf, 0, sizeof(*inf));
        g_launches = 0;
        const int f32 = out_dtype == STPGPU_F32;
        s.beam = s.beam && beam != nullptr;
        switch (precision) {
        case STPGPU_FP64:
            run_imager<double, 0>(c, s, image_size, pars->gridding_correction, dv, vc64, dw, duvw, n_vis, dimg, dbeam,
                f32, inf, device_ptrs != 0);
            break;
        case STPGPU_FP32:
            run_imager<float, 0>(c, s, image_size, pars->gridding_correction, dv, vc64, dw, duvw, n_vis, dimg, dbeam,
                f32, inf, device_ptrs != 0);
            break;
        case STPGPU_FP32C:
            run_imager<float, 1>(c, s, image_size, pars->gridding_correction, dv, vc64, dw, duvw, n_vis, dimg, dbeam,
                f32, inf, device_ptrs != 0);
            break;
        default:
            fail(STPGPU_ERR_INVALID_ARG, "precision");
        }
        if (!device_ptrs && inf->image_size > 0) {
            STPGPU_CUDA_TRY(cudaMemcpyAsync(image, dimg, obytes * npix, cudaMemcpyDeviceToHost, c->stream));
            if (dbeam)
                STPGPU_CUDA_TRY(cudaMemcpyAsync(beam, dbeam, obytes * npix, cudaMemcpyDeviceToHost, c->stream));
        }
        if (timed)
            STPGPU_CUDA_TRY(cudaEventRecord(c->ev1, c->stream));
        STPGPU_CUDA_TRY(cudaStreamSynchronize(c->stream));
        if (timed) {
            float ms = 0.f;
            STPGPU_CUDA_TRY(cudaEventElapsedTime(&ms, c->ev0, c->ev1));
            inf->device_ms = ms;
        }
        inf->n_launches = g_launches;
    });
}

stpgpu_status stpgpu_image_batch(stpgpu_context* c, const stpgpu_snapshot* snapshots, int32_t n_snapshots,
    int precision, int out_dtype, int device_ptrs, stpgpu_imager_info* infos, stpgpu_batch_info* batch_info)
{
    return guard(c, [&] {
        if (!snapshots || n_snapshots <= 0)
            fail(STPGPU_ERR_INVALID_ARG, "empty batch");
        if (out_dtype != STPGPU_F64 && out_dtype != STPGPU_F32)
            fail(STPGPU_ERR_INVALID_ARG, "out_dtype");
        const int f32 = out_dtype == STPGPU_F32;
        switch (precision) {
        case STPGPU_FP64:
            run_batch<double, 0>(c, snapshots, n_snapshots, precision, f32, device_ptrs, infos, batch_info);
            break;
        case STPGPU_FP32:
            run_batch<float, 0>(c, snapshots, n_snapshots, precision, f32, device_ptrs, infos, batch_info);
            break;
        case STPGPU_FP32C:
            run_batch<float, 1>(c, snapshots, n_snapshots, precision, f32, device_ptrs, infos, batch_info);
            break;
        default:
            fail(STPGPU_ERR_INVALID_ARG, "precision");
        }
    });
}

stpgpu_status stpgpu_model_visibilities(stpgpu_context* c, const double* skymodel, int32_t n_src, const double* uvw,
    int64_t n_vis, const double* vis_in, double* vis_out, int device_ptrs)
{
    return guard(c, [&] {
        if (n_src < 0 || n_vis < 0 || (n_vis > 0 && (!uvw || !vis_out)) || (n_src > 0 && !skymodel))
            fail(STPGPU_ERR_INVALID_ARG, "null buffer or negative size");
        if (n_vis == 0)
            return;
        cudaStream_t st = c->stream;
        const double* dsky = skymodel;
        const double* duvw = uvw;
        const double* dvin = vis_in;
        double* dout = vis_out;
        if (!device_ptrs) {
            dsky = to_device<double>(c, "mv_sky", skymodel, 3 * size_t(n_src));
            duvw = to_device<double>(c, "mv_uvw", uvw, 3 * size_t(n_vis));
            if (vis_in)
                dvin = to_device<double>(c, "mv_in", vis_in, 2 * size_t(n_vis));
            dout = c->buf<double>("mv_out", 2 * size_t(n_vis));
        }
        k_model_vis<<<grid1d(n_vis, VIS_THREADS), VIS_THREADS, 0, st>>>(dsky, n_src, duvw, n_vis, dvin,
            vis_in != nullptr, dout);
        STPGPU_CHECK_LAUNCH();
        if (!device_ptrs)
            STPGPU_CUDA_TRY(cudaMemcpyAsync(vis_out, dout, 2 * sizeof(double) * size_t(n_vis), cudaMemcpyDeviceToHost, st));
        STPGPU_CUDA_TRY(cudaStreamSynchronize(st));
    });
}

stpgpu_status stpgpu_set_timing(stpgpu_context* c, int enable)
{
    return guard(c, [&] {
        if (enable)
            for (auto& e : c->pev)
                if (!e)
                    STPGPU_CUDA_TRY(cudaEventCreate(&e));
        c->timing = enable != 0;
    });
}

stpgpu_status stpgpu_image_visibilities(stpgpu_context* c, const double* vis, const double* weights, const double* uvw,
    int64_t n_vis, const stpgpu_imager_pars* pars, const stpgpu_wproj_pars* wproj, const stpgpu_aproj_pars* aproj,
    double* image, double* beam, stpgpu_imager_info* info)
{
    return stpgpu_image_visibilities_ex(c, vis, STPGPU_C128, weights, uvw, n_vis, pars, wproj, aproj, STPGPU_FP64,
        image, beam, STPGPU_F64, 0, info);
}

stpgpu_status stpgpu_convolve_to_grid(stpgpu_context* c, int kernel_function, double kernel_trunc, int support,
    int image_size, const double* uv, const double* vis, const double* weights, int64_t n_vis, int kernel_exact,
    int oversampling, int shift_uv, int halfplane, int generate_beam, const stpgpu_wproj_pars* wproj, const double* w,
    double cell_size, int analytic_gcf, double* vis_grid, double* sampling_grid, double* sample_grid_total)
{
    return guard(c, [&] {
        if (kernel_function < 0 || kernel_function > 5)
            fail(STPGPU_ERR_INVALID_ARG, "unknown kernel function");
        if (n_vis < 0 || (n_vis > 0 && (!uv || !vis || !weights)) || !vis_grid)
            fail(STPGPU_ERR_INVALID_ARG, "null buffer");
        ImagerSetup s;
        s.kf = kernel_function;
        s.trunc = kernel_trunc;
        s.support = support;
        s.N = image_size;
        s.kernel_exact = kernel_exact;
        s.os = oversampling;
        s.shift_uv = shift_uv;
        s.halfplane = halfplane;
        s.beam = generate_beam && sampling_grid;
        s.analytic = analytic_gcf;
        s.cell_size = cell_size;
        const bool wp = wproj && wproj->num_wplanes > 0;
        if (wp) {
            if (!w)
                fail(STPGPU_ERR_INVALID_ARG, "W-projection needs w");
            if (!(cell_size > 0.0))
                fail(STPGPU_ERR_INVALID_ARG, "W-projection needs cell_size > 0");
            s.nplanes = wproj->num_wplanes;
            s.max_support = wproj->max_wpconv_support;
            s.undersampling = wproj->undersampling_opt;
            s.trunc_perc = wproj->kernel_trunc_perc;
            s.wmedian = wproj->wplanes_median;
            if (wproj->hankel_opt) {
                if (wproj->interp_type < 0 || wproj->interp_type > 2)
                    fail(STPGPU_ERR_INVALID_ARG, "unknown interp_type");
                s.hankel = 1;
                s.proj_slice = wproj->hankel_proj_slice ? 1 : 0;
                s.cubic = wproj->interp_type == 1;
            }
        }
        if (!kernel_exact && !wp && oversampling < 1)
            fail(STPGPU_ERR_INVALID_ARG, "oversampling must be >= 1");
        // uv (n x 2) [+ w] in pixels as an n x 3 device array
        double* duv = c->buf<double>("in_uv", 3 * size_t(std::max<int64_t>(n_vis, 1)));
        if (n_vis) {
            STPGPU_CUDA_TRY(cudaMemcpyAsync(duv, uv, sizeof(double) * 2 * n_vis, cudaMemcpyHostToDevice, c->stream));
            if (wp)
                STPGPU_CUDA_TRY(
                    cudaMemcpyAsync(duv + 2 * n_vis, w, sizeof(double) * n_vis, cudaMemcpyHostToDevice, c->stream));
        }
        const double* dvis = to_device<double>(c, "in_vis", vis, 2 * size_t(n_vis));
        const double* dw = to_device<double>(c, "in_w", weights, size_t(n_vis));
        c->drop_single(); // this call reuses the imager's buffers
        GridOut g = run_gridder<double, 0>(c, s, dvis, 0, dw, duv, 1, n_vis);
        ScalarPack sb = read_back(c, g, false);
        if (sb.err & 4u) { // redo with the 64-bit |w| sort
            s.full_wsort = 1;
            g = run_gridder<double, 0>(c, s, dvis, 0, dw, duv, 1, n_vis);
            sb = read_back(c, g, false);
        }
        const size_t cells = size_t(g.image_rows) * size_t(image_size);
        STPGPU_CUDA_TRY(cudaMemcpyAsync(vis_grid, g.grid, sizeof(double2) * cells, cudaMemcpyDeviceToHost, c->stream));
        if (s.beam)
            STPGPU_CUDA_TRY(
                cudaMemcpyAsync(sampling_grid, g.beam, sizeof(double2) * cells, cudaMemcpyDeviceToHost, c->stream));
        STPGPU_CUDA_TRY(cudaStreamSynchronize(c->stream));
        if (sample_grid_total)
            *sample_grid_total = sb.total;
    });
}

stpgpu_status stpgpu_source_find_ex(stpgpu_context* c, const void* image, int image_dtype, int32_t rows, int32_t cols,
    const stpgpu_sf_pars* pars, int32_t* label_map, int device_ptrs, stpgpu_island* islands, int32_t capacity,
    int32_t* n_islands, stpgpu_sf_info* info)
{
    return guard(c, [&] {
        if (!image || !pars || !n_islands)
            fail(STPGPU_ERR_INVALID_ARG, "null argument");
        if (image_dtype != STPGPU_F64 && image_dtype != STPGPU_F32)
            fail(STPGPU_ERR_INVALID_ARG, "image_dtype");
        const int64_t n = int64_t(rows) * cols;
        const size_t eb = image_dtype == STPGPU_F32 ? 4 : 8;
        if (!device_ptrs)
            STPGPU_CUDA_TRY(cudaEventRecord(c->ev0, c->stream));
        const void* dimg = image;
        if (!device_ptrs && n > 0)
            dimg = to_device<unsigned char>(c, "sf_in", image, eb * size_t(n));
        int32_t* dl = device_ptrs ? label_map : nullptr;
        std::vector<stpgpu_island> isl;
        stpgpu_sf_info local {};
        stpgpu_sf_info* inf = info ? info : &local;
        std::memset(inf, 0, sizeof(*inf));
        const bool want = label_map != nullptr;
        if (image_dtype == STPGPU_F32)
            run_source_find<float>(c, reinterpret_cast<const float*>(dimg), rows, cols, *pars, dl, want, isl, *inf);
        else
            run_source_find<double>(c, reinterpret_cast<const double*>(dimg), rows, cols, *pars, dl, want, isl, *inf);
        if (!device_ptrs && label_map) {
            const int32_t* src = c->buf<int32_t>("ccl_L", n);
            STPGPU_CUDA_TRY(cudaMemcpyAsync(label_map, src, sizeof(int32_t) * n, cudaMemcpyDeviceToHost, c->stream));
        }
        if (!device_ptrs)
            STPGPU_CUDA_TRY(cudaEventRecord(c->ev1, c->stream));
        STPGPU_CUDA_TRY(cudaStreamSynchronize(c->stream));
        if (!device_ptrs) {
            float ms = 0.f;
            STPGPU_CUDA_TRY(cudaEventElapsedTime(&ms, c->ev0, c->ev1));
            inf->device_ms = ms;
        }
        *n_islands = int32_t(isl.size());
        if (int32_t(isl.size()) > capacity)
            fail(STPGPU_ERR_CAPACITY, "island buffer too small: need " + std::to_string(isl.size()));
        if (!isl.empty())
            std::memcpy(islands, isl.data(), sizeof(stpgpu_island) * isl.size());
    });
}

stpgpu_status stpgpu_source_find(stpgpu_context* c, const double* image, int32_t rows, int32_t cols,
    const stpgpu_sf_pars* pars, int32_t* label_map, stpgpu_island* islands, int32_t capacity, int32_t* n_islands,
    stpgpu_sf_info* info)
{
    return stpgpu_source_find_ex(c, image, STPGPU_F64, rows, cols, pars, label_map, 0, islands, capacity, n_islands,
        info);
}

} // extern "C"

// ------------------------------------------------------------------ serving

namespace {

struct ServerJob {
    int64_t ticket = 0;
    stpgpu_request req {};
    stpgpu_result res {};
    bool done = false;
};

// Device working set of one request (inputs, items, binned entries, W-planes and
// W-kernel tables, grid, FFT output, image, source-finder arrays), bytes.
int64_t request_bytes(const ImagerSetup& s, int image_size, int64_t n, int vis_c64, int precision, int find_sources,
    int correction)
{
    const int64_t rb = precision == STPGPU_FP64 ? 8 : 4;
    const int64_t N = s.N, rows = N / 2 + 1;
    const int conv = s.nplanes > 0 ? s.max_support : s.support;
    int64_t b = n * ((vis_c64 ? 8 : 16) + 8 + 24) + n * (rb == 8 ? 48 : 32); // items: 48 / 32 B records
    b += int64_t(entry_capacity(s.N, 2 * conv + 1, n)) * (rb == 8 ? 32 : 16); // entry records
    b += std::max<int64_t>(n, 1) * kEntrySlots * 4;                           // their places in the bins
    b += 12 * (rows / kBlk + 40) * (N / kBlk + 40);                           // bins
    if (s.kernel_exact)
        b += n * (2 * 8 + 2 * 8 * (2 * conv + 1)); // fractional positions, 1-D kernels
    if (s.nplanes > 0) {
        b += n * (rb == 8 ? 48 : 32); // items in |w| order
        const int64_t os = std::max(1, (s.os >> 1) << 1), cs = (os / 2) * 2 + 1, K = 2 * conv + 1;
        const WkShape ks = wk_shape(s, int(os));
        b += n * 55; // |w| sort (CUB's own buffers with it), planes
        b += int64_t(s.nplanes) * (cs * cs * K * K * 2 * rb + int64_t(ks.lh) * ks.lh * 16);
        b += int64_t(ks.q_cells + ks.t_cells) * 16 + (ks.workarea + ks.arr) * 8;
        if (s.hankel && !ks.too_large())
            b += int64_t(s.nplanes) * (ks.half * 16 + ks.arr * 48); // radial profiles, transforms, spline
    }
    b += rows * N * 2 * rb + N * N * rb + int64_t(image_size) * image_size * rb;
    if (precision == STPGPU_FP32C && wide_fft_needed(s, image_size, correction))
        b += rows * N * 2 * rb + N * N * rb; // double-precision grid and c2r output
    if (find_sources) // classes, parents, ranks, labels, foreground list; at worst list arrays (20 B) for every
                      // pixel and per-label arrays (160 B) for every second pixel
        b += int64_t(image_size) * image_size * (1 + 4 + 4 + 4 + 4 + 20 + 80 + 2) + (int64_t(8) << 20); // + clip lists
    return b + (int64_t(8) << 20);
}

// One request on one slot context (host buffers in and out).
template <typename R, int COMP>
void serve_request(stpgpu_context* c, const stpgpu_request& r, stpgpu_result& res)
{
    int image_size = 0;
    ImagerSetup s = setup_from(&r.pars, &r.wproj, nullptr, image_size);
    s.beam = 0;
    const int c64 = r.vis_dtype == STPGPU_C64;
    const int f32 = r.out_dtype == STPGPU_F32;
    const int64_t n = r.n_vis;
    const void* dv = to_device<unsigned char>(c, "in_vis", r.vis, (c64 ? 8 : 16) * size_t(n));
    const double* dw = to_device<double>(c, "in_w", r.weights, size_t(n));
    const double* duvw = to_device<double>(c, "in_uvw", r.uvw, 3 * size_t(n));
    const int64_t npix = int64_t(image_size) * image_size;
    const size_t ob = f32 ? 4 : 8;
    void* dimg = c->buf<unsigned char>("srv_img", ob * size_t(std::max<int64_t>(npix, 1)));
    const auto t_in = std::chrono::steady_clock::now();
    run_imager<R, COMP>(c, s, image_size, r.pars.gridding_correction, dv, c64, dw, duvw, n, dimg, nullptr, f32,
        &res.imager);
    const auto t_img = std::chrono::steady_clock::now();
    if (res.imager.image_size > 0) {
        if (r.image)
            STPGPU_CUDA_TRY(cudaMemcpyAsync(r.image, dimg, ob * npix, cudaMemcpyDeviceToHost, c->stream));
        if (r.find_sources) {
            std::vector<stpgpu_island> isl;
            if (f32)
                run_source_find<float>(c, reinterpret_cast<const float*>(dimg), image_size, image_size, r.sf, nullptr,
                    r.label_map != nullptr, isl, res.sf);
            else
                run_source_find<double>(c, reinterpret_cast<const double*>(dimg), image_size, image_size, r.sf,
                    nullptr, r.label_map != nullptr, isl, res.sf);
            if (r.label_map)
                STPGPU_CUDA_TRY(cudaMemcpyAsync(r.label_map, c->buf<int32_t>("ccl_L", npix), sizeof(int32_t) * npix,
                    cudaMemcpyDeviceToHost, c->stream));
            res.n_islands = int32_t(isl.size());
            if (int32_t(isl.size()) > r.island_capacity)
                fail(STPGPU_ERR_CAPACITY, "island buffer too small: need " + std::to_string(isl.size()));
            if (!isl.empty())
                std::memcpy(r.islands, isl.data(), sizeof(stpgpu_island) * isl.size());
        }
    }
    STPGPU_CUDA_TRY(cudaStreamSynchronize(c->stream));
    // STPGPU_LOG_SLOW=<ms>: host-side phase times of requests slower than that
    static const char* slow = std::getenv("STPGPU_LOG_SLOW");
    if (slow) {
        const auto t_end = std::chrono::steady_clock::now();
        auto ms = [](auto a, auto b) { return std::chrono::duration<double, std::milli>(b - a).count(); };
        if (ms(t_in, t_end) > std::atof(slow))
            std::fprintf(stderr, "stpgpu slow request: N=%d n_vis=%lld imager %.3f ms, source finder %.3f ms\n",
                image_size, (long long)n, ms(t_in, t_img), ms(t_img, t_end));
    }
}

} // namespace

struct stpgpu_server {
    stpgpu_server_pars pars {};
    std::vector<stpgpu_context*> slots;
    std::vector<std::thread> workers;
    std::mutex mu;
    std::condition_variable cv_work, cv_done;
    std::deque<ServerJob*> queue;
    std::unordered_map<int64_t, std::unique_ptr<ServerJob>> jobs;
    int64_t next_ticket = 1;
    int64_t inflight = 0, inflight_bytes = 0;
    bool stop = false;
    int paused = 0; // stpgpu_server_prepare holds the slots: no admission
    std::chrono::steady_clock::time_point t0;
    std::vector<double> latency_ms;
    double first_submit = -1.0, last_done = 0.0;
    stpgpu_server_stats st {};

    double now_ms() const
    {
        return std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
    }

    void worker(int k)
    {
        stpgpu_context* c = slots[k];
        cudaSetDevice(c->device);
        for (;;) {
            ServerJob* job = nullptr;
            {
                std::unique_lock<std::mutex> lk(mu);
                // first-in first-out: the head starts once its working set fits
                auto admissible = [&] {
                    return !paused && !queue.empty()
                        && inflight_bytes + queue.front()->res.est_bytes <= pars.hbm_budget_bytes;
                };
                cv_work.wait(lk, [&] { return stop || admissible(); });
                if (queue.empty() && stop)
                    return;
                if (!admissible())
                    continue;
                job = queue.front();
                queue.pop_front();
                inflight++;
                inflight_bytes += job->res.est_bytes;
                st.peak_in_flight = std::max(st.peak_in_flight, inflight);
                st.peak_admitted_bytes = std::max(st.peak_admitted_bytes, inflight_bytes);
                job->res.admit_ms = now_ms();
            }
            const stpgpu_status status = guard(c, [&] {
                g_launches = 0;
                switch (pars.precision) {
                case STPGPU_FP64:
                    serve_request<double, 0>(c, job->req, job->res);
                    break;
                case STPGPU_FP32:
                    serve_request<float, 0>(c, job->req, job->res);
                    break;
                default:
                    serve_request<float, 1>(c, job->req, job->res);
                    break;
                }
            });
            {
                std::lock_guard<std::mutex> lk(mu);
                job->res.status = status;
                if (status != STPGPU_OK)
                    std::snprintf(job->res.error, sizeof(job->res.error), "%s", c->err.c_str());
                job->res.done_ms = now_ms();
                job->done = true;
                inflight--;
                inflight_bytes -= job->res.est_bytes;
                if (status == STPGPU_OK) {
                    st.completed++;
                    latency_ms.push_back(job->res.done_ms - job->res.submit_ms);
                    last_done = std::max(last_done, job->res.done_ms);
                } else {
                    st.failed++;
                }
            }
            cv_done.notify_all();
            cv_work.notify_all();
        }
    }
};

extern "C" {

stpgpu_status stpgpu_server_create(const stpgpu_server_pars* pars, stpgpu_server** out)
{
    if (!pars || !out || pars->slots < 1 || pars->hbm_budget_bytes <= 0)
        return STPGPU_ERR_INVALID_ARG;
    if (pars->precision < STPGPU_FP64 || pars->precision > STPGPU_FP32C)
        return STPGPU_ERR_INVALID_ARG;
    *out = nullptr;
    auto* sv = new stpgpu_server();
    sv->pars = *pars;
    sv->t0 = std::chrono::steady_clock::now();
    for (int k = 0; k < pars->slots; k++) {
        stpgpu_context* c = nullptr;
        const stpgpu_status s = stpgpu_create(pars->device, &c);
        if (s != STPGPU_OK) {
            for (auto x : sv->slots)
                stpgpu_destroy(x);
            delete sv;
            return s;
        }
        sv->slots.push_back(c);
    }
    for (int k = 0; k < pars->slots; k++)
        sv->workers.emplace_back([sv, k] { sv->worker(k); });
    *out = sv;
    return STPGPU_OK;
}

stpgpu_status stpgpu_server_destroy(stpgpu_server* sv)
{
    if (!sv)
        return STPGPU_OK;
    {
        std::unique_lock<std::mutex> lk(sv->mu);
        sv->cv_done.wait(lk, [&] { return sv->queue.empty() && sv->inflight == 0; });
        sv->stop = true;
    }
    sv->cv_work.notify_all();
    for (auto& t : sv->workers)
        t.join();
    for (auto c : sv->slots)
        stpgpu_destroy(c);
    delete sv;
    return STPGPU_OK;
}

namespace {

// Parameter checks of a request and its working-set estimate.
stpgpu_status check_request(const stpgpu_server* sv, const stpgpu_request* r, int64_t& est)
{
    est = 0;
    try {
        int image_size = 0;
        ImagerSetup s = setup_from(&r->pars, &r->wproj, nullptr, image_size);
        if (r->pars.generate_beam)
            return STPGPU_ERR_UNSUPPORTED;
        if (image_size <= 0 || image_size > s.N || (image_size % 2) != 0)
            return STPGPU_ERR_INVALID_ARG;
        if (r->n_vis < 0 || (r->n_vis > 0 && (!r->vis || !r->weights || !r->uvw)) || (!r->image && !r->find_sources))
            return STPGPU_ERR_INVALID_ARG;
        if ((r->vis_dtype != STPGPU_C128 && r->vis_dtype != STPGPU_C64)
            || (r->out_dtype != STPGPU_F64 && r->out_dtype != STPGPU_F32))
            return STPGPU_ERR_INVALID_ARG;
        if (r->find_sources && (r->island_capacity < 0 || (r->island_capacity > 0 && !r->islands)))
            return STPGPU_ERR_INVALID_ARG;
        est = request_bytes(s, image_size, r->n_vis, r->vis_dtype == STPGPU_C64, sv->pars.precision, r->find_sources,
            r->pars.gridding_correction);
    } catch (const Error& e) {
        return e.status;
    }
    if (est > sv->pars.hbm_budget_bytes)
        return STPGPU_ERR_OOM;
    return STPGPU_OK;
}

} // namespace

stpgpu_status stpgpu_server_submit(stpgpu_server* sv, const stpgpu_request* r, int64_t* ticket)
{
    if (!sv || !r || !ticket)
        return STPGPU_ERR_INVALID_ARG;
    int64_t est = 0;
    if (const stpgpu_status bad = check_request(sv, r, est))
        return bad;
    auto job = std::make_unique<ServerJob>();
    job->req = *r;
    job->res.est_bytes = est;
    {
        std::lock_guard<std::mutex> lk(sv->mu);
        job->ticket = sv->next_ticket++;
        job->res.submit_ms = sv->now_ms();
        if (sv->first_submit < 0)
            sv->first_submit = job->res.submit_ms;
        sv->st.submitted++;
        *ticket = job->ticket;
        sv->queue.push_back(job.get());
        sv->jobs[job->ticket] = std::move(job);
    }
    sv->cv_work.notify_all();
    return STPGPU_OK;
}

stpgpu_status stpgpu_server_prepare(stpgpu_server* sv, const stpgpu_request* r, stpgpu_result* out)
{
    if (!sv || !r)
        return STPGPU_ERR_INVALID_ARG;
    stpgpu_result res {};
    if (const stpgpu_status bad = check_request(sv, r, res.est_bytes))
        return bad;
    {
        // hold admission and let the requests in flight finish: the slots'
        // contexts are then free for this thread
        std::unique_lock<std::mutex> lk(sv->mu);
        sv->paused++;
        sv->cv_done.wait(lk, [&] { return sv->inflight == 0; });
    }
    stpgpu_status status = STPGPU_OK;
    for (stpgpu_context* c : sv->slots) {
        cudaSetDevice(c->device);
        res = stpgpu_result {};
        status = guard(c, [&] {
            switch (sv->pars.precision) {
            case STPGPU_FP64:
                serve_request<double, 0>(c, *r, res);
                break;
            case STPGPU_FP32:
                serve_request<float, 0>(c, *r, res);
                break;
            default:
                serve_request<float, 1>(c, *r, res);
                break;
            }
        });
        if (status != STPGPU_OK) {
            std::snprintf(res.error, sizeof(res.error), "%s", c->err.c_str());
            break;
        }
    }
    res.status = status;
    if (out)
        *out = res;
    {
        std::lock_guard<std::mutex> lk(sv->mu);
        sv->paused--;
    }
    sv->cv_work.notify_all();
    return status;
}

stpgpu_status stpgpu_server_wait(stpgpu_server* sv, int64_t ticket, double timeout_s, stpgpu_result* out)
{
    if (!sv)
        return STPGPU_ERR_INVALID_ARG;
    std::unique_lock<std::mutex> lk(sv->mu);
    auto it = sv->jobs.find(ticket);
    if (it == sv->jobs.end())
        return STPGPU_ERR_INVALID_ARG;
    ServerJob* job = it->second.get();
    if (timeout_s < 0)
        sv->cv_done.wait(lk, [&] { return job->done; });
    else if (!sv->cv_done.wait_for(lk, std::chrono::duration<double>(timeout_s), [&] { return job->done; }))
        return STPGPU_ERR_TIMEOUT;
    if (out)
        *out = job->res;
    const stpgpu_status s = stpgpu_status(job->res.status);
    sv->jobs.erase(it);
    return s;
}

stpgpu_status stpgpu_server_stats_get(stpgpu_server* sv, stpgpu_server_stats* out)
{
    if (!sv || !out)
        return STPGPU_ERR_INVALID_ARG;
    std::lock_guard<std::mutex> lk(sv->mu);
    stpgpu_server_stats s = sv->st;
    s.in_flight = sv->inflight;
    s.queued = int64_t(sv->queue.size());
    std::vector<double> l = sv->latency_ms;
    if (!l.empty()) {
        std::sort(l.begin(), l.end());
        auto pct = [&](double q) {
            const double pos = q * double(l.size() - 1);
            const size_t i = size_t(pos);
            const double f = pos - double(i);
            return i + 1 < l.size() ? l[i] * (1.0 - f) + l[i + 1] * f : l[i];
        };
        s.p50_ms = pct(0.50);
        s.p99_ms = pct(0.99);
        double sum = 0.0;
        for (double v : l)
            sum += v;
        s.mean_ms = sum / double(l.size());
        const double span = sv->last_done - sv->first_submit;
        s.throughput_rps = span > 0 ? double(s.completed) / (span / 1e3) : 0.0;
    }
    *out = s;
    return STPGPU_OK;
}

} // extern "C"

// ------------------------------------------------------- allocation-free labelling
//
// stpgpu_label_noalloc runs the connected-component labeller (k_ccl_* above)
// with its working arrays in one file-scope device array instead of
// context-owned buffers.  It exists for callers that must not allocate:
//  * a real-time detection stage that runs between the imaging launches of a
//    stream-ordered pipeline: cudaMalloc/cudaFree synchronise the whole device
//    and would stall the imaging streams that share it, breaking the snapshot
//    cadence;
//  * a process whose device memory is already owned by another allocator (a
//    caching allocator or a memory pool that reserved the free HBM up front),
//    where an allocation by this library could fail with out-of-memory in the
//    middle of a run;
// neither can create a stpgpu_context, which allocates its buffers, stream and
// events.  The call makes no cudaMalloc, cudaFree or allocating library call;
// host-side it uses no heap either (no exceptions, strings or containers).
//
// Scratch layout for n = rows * cols pixels (byte offsets, 256-aligned):
//   cls  nchunks * CCL_CHUNK bytes   pixel class (0 background, 1 positive,
//                       2 negative), background padding past n
//   P    n uint32       union-find parents
//   R    n uint32       final label number of each root
//   misc 8 uint32       row totals and the union-find step-bound flag; the
//                       flag MUST start at zero, so every call clears misc
//                       before the first kernel
//   cnt, off            3 * (nchunks + 1) uint32 each: positive roots,
//                       negative roots and foreground keys per chunk of
//                       CCL_CHUNK keys, and their exclusive scans
// Everything except misc is fully written before it is read in each call.
// The array is shared by every call on a device: two calls whose kernels
// overlap on the GPU (different streams, or different host threads) race on
// it and give wrong labels.  The first call on a device resolves the array's
// device address (cudaGetSymbolAddress, that device current) and caches it;
// that first call should come before any stream capture.

namespace stpgpu {

constexpr size_t noalloc_align(size_t b) { return (b + 255) / 256 * 256; }
constexpr size_t noalloc_chunks(size_t n) { return (n + CCL_CHUNK - 1) / CCL_CHUNK; }
constexpr size_t noalloc_bytes(size_t n)
{
    return noalloc_align(noalloc_chunks(n) * CCL_CHUNK) + 2 * noalloc_align(4 * n) + 256
        + 2 * noalloc_align(12 * (noalloc_chunks(n) + 1));
}
constexpr size_t kNoallocScratchBytes = noalloc_bytes(STPGPU_NOALLOC_MAX_PIXELS);

static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoallocScratchBytes];

constexpr int kNoallocMaxDevices = 64;
static std::mutex g_noalloc_mu;
static unsigned char* g_noalloc_ptr[kNoallocMaxDevices] = {};

static stpgpu_status noalloc_msg(char* buf, size_t len, stpgpu_status s, const char* what, cudaError_t e)
{
    if (buf && len)
        std::snprintf(buf, len, "%s%s%s", what, e == cudaSuccess ? "" : ": ",
            e == cudaSuccess ? "" : cudaGetErrorString(e));
    return s;
}

template <typename T>
static cudaError_t noalloc_label_run(unsigned char* base, cudaStream_t st, const T* img, int rows, int cols,
    double tp, double tn, int findneg, int conn4, int slice, int32_t* L, uint32_t* h)
{
    const int64_t n = int64_t(rows) * cols;
    const size_t nch = noalloc_chunks(size_t(n));
    size_t o = 0;
    CclBufs b;
    b.cls = base + o;
    o += noalloc_align(nch * CCL_CHUNK);
    b.P = reinterpret_cast<uint32_t*>(base + o);
    o += noalloc_align(4 * size_t(n));
    b.R = reinterpret_cast<uint32_t*>(base + o);
    o += noalloc_align(4 * size_t(n));
    b.misc = reinterpret_cast<uint32_t*>(base + o);
    o += 256;
    b.cnt = reinterpret_cast<uint32_t*>(base + o);
    o += noalloc_align(12 * (nch + 1));
    b.off = reinterpret_cast<uint32_t*>(base + o);
    b.fgl = nullptr;
    b.L = L;
    cudaError_t e = cudaMemsetAsync(b.misc, 0, 8 * sizeof(uint32_t), st);
    if (e != cudaSuccess)
        return e;
    const CclGeom geom { rows, cols, rows / 2, cols / 2 };
    if ((e = ccl_enqueue<T>(st, img, geom, nullptr, tp, tn, findneg, conn4, slice, b)) != cudaSuccess)
        return e;
    // label counts and the step-bound flag, read back into host stack memory
    if ((e = cudaMemcpyAsync(h, b.misc, 4 * sizeof(uint32_t), cudaMemcpyDeviceToHost, st)) != cudaSuccess)
        return e;
    return cudaStreamSynchronize(st);
}

} // namespace stpgpu

extern "C" stpgpu_status stpgpu_label_noalloc(int device, void* stream, const void* image, int image_dtype,
    int32_t rows, int32_t cols, double analysis_thresh_pos, double analysis_thresh_neg, int find_negative_sources,
    int ccl_4connectivity, int ccl_slice_cols, int32_t* label_map, int32_t* n_labels_pos, int32_t* n_labels_neg,
    char* err_msg, size_t err_msg_len)
{
    using namespace stpgpu;
    if (err_msg && err_msg_len)
        err_msg[0] = '\0';
    if (!image || !label_map)
        return noalloc_msg(err_msg, err_msg_len, STPGPU_ERR_INVALID_ARG, "null image or label_map", cudaSuccess);
    if (image_dtype != STPGPU_F64 && image_dtype != STPGPU_F32)
        return noalloc_msg(err_msg, err_msg_len, STPGPU_ERR_INVALID_ARG, "image_dtype", cudaSuccess);
    if (rows <= 0 || cols <= 0 || (rows % 2) || (cols % 2) || rows > 65536 || cols > 65536)
        return noalloc_msg(err_msg, err_msg_len, STPGPU_ERR_INVALID_ARG,
            "image dimensions must be positive, even and at most 65536 (ccl.h:116-119)", cudaSuccess);
    if (int64_t(rows) * cols > int64_t(STPGPU_NOALLOC_MAX_PIXELS)) {
        if (err_msg && err_msg_len)
            std::snprintf(err_msg, err_msg_len,
                "image of %lld pixels exceeds the allocation-free labeller's maximum of %lld pixels",
                (long long)(int64_t(rows) * cols), (long long)STPGPU_NOALLOC_MAX_PIXELS);
        return STPGPU_ERR_INVALID_ARG;
    }
    if (device < 0 || device >= kNoallocMaxDevices)
        return noalloc_msg(err_msg, err_msg_len, STPGPU_ERR_INVALID_ARG, "device ordinal", cudaSuccess);
    int prev = 0;
    cudaError_t e = cudaGetDevice(&prev);
    if (e != cudaSuccess)
        return noalloc_msg(err_msg, err_msg_len, STPGPU_ERR_NO_DEVICE, "cudaGetDevice", e);
    if ((e = cudaSetDevice(device)) != cudaSuccess)
        return noalloc_msg(err_msg, err_msg_len, STPGPU_ERR_NO_DEVICE, "cudaSetDevice", e);
    unsigned char* base = nullptr;
    {
        // set-up, once per device, with that device current
        std::lock_guard<std::mutex> lk(g_noalloc_mu);
        if (!g_noalloc_ptr[device]) {
            void* p = nullptr;
            e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
            if (e != cudaSuccess) {
                cudaSetDevice(prev);
                return noalloc_msg(err_msg, err_msg_len, STPGPU_ERR_CUDA, "cudaGetSymbolAddress(scratch)", e);
            }
            g_noalloc_ptr[device] = static_cast<unsigned char*>(p);
        }
        base = g_noalloc_ptr[device];
    }
    const int slice = ccl_slice_cols > 0 ? ccl_slice_cols : std::max(2, cols / 8);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    uint32_t h[4] = { 0, 0, 0, 0 }; // positive labels, negative labels, foreground keys, step-bound flag
    if (image_dtype == STPGPU_F32)
        e = noalloc_label_run<float>(base, st, static_cast<const float*>(image), rows, cols, analysis_thresh_pos,
            analysis_thresh_neg, find_negative_sources, ccl_4connectivity, slice, label_map, h);
    else
        e = noalloc_label_run<double>(base, st, static_cast<const double*>(image), rows, cols, analysis_thresh_pos,
            analysis_thresh_neg, find_negative_sources, ccl_4connectivity, slice, label_map, h);
    cudaSetDevice(prev);
    if (e != cudaSuccess)
        return noalloc_msg(err_msg, err_msg_len, STPGPU_ERR_CUDA, "labelling", e);
    if (h[3])
        return noalloc_msg(err_msg, err_msg_len, STPGPU_ERR_DEVICE, "labeler gave up (union-find step bound)",
            cudaSuccess);
    if (n_labels_pos)
        *n_labels_pos = int32_t(h[0]);
    if (n_labels_neg)
        *n_labels_neg = int32_t(h[1]);
    return STPGPU_OK;
}
