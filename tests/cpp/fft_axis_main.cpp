// The passes along the columns (k_fft_axis) on the CPU: no block reads a cell
// that another block of the same pass writes (the passes work in place and
// blocks are not ordered), and two passes are the backward transform.
#include "fft_kernels.cuh"

#include <algorithm>
#include <complex>

namespace stpgpu {

struct Cell;
static const Cell* g_begin = nullptr;
static const Cell* g_end = nullptr;
static std::mutex g_mutex;
static std::vector<std::pair<size_t, unsigned>> g_reads, g_writes; // cell, block

static void note(std::vector<std::pair<size_t, unsigned>>& log, const Cell* p);

struct Cell {
    double x = 0.0, y = 0.0;
    Cell() = default;
    Cell(const Cell& o)
        : x(o.x)
        , y(o.y)
    {
        note(g_reads, &o);
    }
    Cell& operator=(const Cell& o)
    {
        note(g_reads, &o);
        note(g_writes, this);
        x = o.x;
        y = o.y;
        return *this;
    }
};

static void note(std::vector<std::pair<size_t, unsigned>>& log, const Cell* p)
{
    if (p < g_begin || p >= g_end)
        return;
    std::lock_guard<std::mutex> lock(g_mutex);
    log.emplace_back(size_t(p - g_begin), blockIdx.y * gridDim.x + blockIdx.x);
}

struct Probe {
    double v;
};
template <>
struct Cplx<Probe> {
    using T = Cell;
};

alignas(16) unsigned char smem_fft[1 << 18];

template <int L, bool FIRST>
int pass(std::vector<Cell>& grid, int ld, int rows, int N, const std::vector<Cell>& tw)
{
    g_reads.clear();
    g_writes.clear();
    launch(Dim3 { unsigned(rows + 31) / 32, unsigned(N / L / axis_groups(L)), 1 }, axis_threads(L),
        [&] { k_fft_axis<Probe, L, FIRST>(grid.data(), ld, rows, N, tw.data()); });
    std::vector<unsigned> writer(grid.size(), ~0u);
    int bad = 0;
    for (auto& w : g_writes) {
        bad += writer[w.first] != ~0u && writer[w.first] != w.second;
        bad += int(w.first % size_t(ld)) >= rows;
        writer[w.first] = w.second;
    }
    for (auto& r : g_reads)
        bad += writer[r.first] != ~0u && writer[r.first] != r.second;
    return bad;
}

template <int L1, int L2>
int check(int N)
{
    const int rows = N / 2 + 1, ld = (rows + 15) / 16 * 16;
    int logm = 0;
    while ((2 << logm) < N)
        logm++;
    std::vector<double2> roots(tw_size(N));
    launch(Dim3 { unsigned(tw_size(N) + 255) / 256, 1, 1 }, 256, [&] { k_fft_tables<double>(N, logm, roots.data()); });
    std::vector<Cell> tw(roots.size()), grid(size_t(ld) * N);
    for (size_t i = 0; i < roots.size(); i++) {
        tw[i].x = roots[i].x;
        tw[i].y = roots[i].y;
    }
    std::vector<std::complex<double>> in(grid.size());
    uint32_t seed = 1;
    for (size_t i = 0; i < grid.size(); i++) {
        seed = seed * 1664525u + 1013904223u;
        grid[i].x = double(seed >> 8) / (1 << 24) - 0.5;
        seed = seed * 1664525u + 1013904223u;
        grid[i].y = double(seed >> 8) / (1 << 24) - 0.5;
        in[i] = { grid[i].x, grid[i].y };
    }
    g_begin = grid.data();
    g_end = grid.data() + grid.size();
    const int a = pass<L1, true>(grid, ld, rows, N, tw), b = pass<L2, false>(grid, ld, rows, N, tw);
    g_begin = g_end = nullptr;
    double err = 0.0;
    for (int k = 0; k < N; k += 7)
        for (int r : { 0, 1, 31, 32, rows - 1 }) {
            std::complex<double> s = 0.0;
            for (int c = 0; c < N; c++)
                s += in[size_t(c) * ld + r] * std::polar(1.0, 2.0 * M_PI * double(int64_t(c) * k % N) / N);
            const Cell& z = grid[size_t(axis_place(k, N)) * ld + r];
            err = std::max(err, std::abs(s - std::complex<double>(z.x, z.y)));
        }
    std::printf("N %d: cells shared by two blocks in pass 1: %d, pass 2: %d; error %.1e\n", N, a, b, err);
    return a + b + (err > 1e-11);
}

} // namespace stpgpu

int main() { return stpgpu::check<16, 16>(256) + stpgpu::check<32, 16>(512) ? 1 : 0; }
