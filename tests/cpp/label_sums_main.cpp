// k_label_sums on the CPU while a label has more pixels than the one-block
// sort takes: their order is not formed yet (the host sorts all of them and
// sums again), so nothing may be read through it.
#include <algorithm>
#include <atomic>

static int g_pixels = 0;
static std::atomic<int> g_outside { 0 };

template <typename T>
double ld(const T* p, int64_t i)
{
    if (i < 0 || i >= g_pixels) {
        g_outside++;
        return 0.0;
    }
    return double(p[i]);
}

#include "label_sums.cuh"

int main()
{
    const int rows = 256, cols = 256;
    g_pixels = rows * cols;
    std::vector<float> img(g_pixels);
    for (int i = 0; i < g_pixels; i++)
        img[i] = float(i % 97) - 20.0f;
    const uint32_t small = 100, large = SEG_BIG + 5;
    const uint32_t misc[3] = { 2, 0, small + large };
    const FgSizes z { misc, 2, small + large };
    // ranges from k_seg_alloc (the split of a range that is not sorted is still zero), pixels from k_seg_sort
    const std::vector<uint32_t> begin = { 0, small }, end = { small, small + large }, listed = { 1, 0 };
    std::vector<uint32_t> split = { small, 0 }, pixels(small + large, 0xfffffff0u);
    const uint32_t nlisted = 2;
    for (uint32_t i = 0; i < small; i++)
        pixels[i] = 3 * i; // all in the left half of the image
    std::vector<double> mom(12);
    std::vector<int> ns(2);
    auto run = [&](uint32_t longest) {
        std::fill(mom.begin(), mom.end(), -1.0);
        launch(Dim3 { 2, 1, 1 }, 32 * kSumWarps, [&] {
            k_label_sums<float>(z, img.data(), rows, cols, pixels.data(), begin.data(), end.data(), split.data(),
                listed.data(), &nlisted, longest, mom.data(), ns.data());
        });
    };
    int bad = 0;
    auto check = [&](int l) {
        double v = 0.0, x = 0.0;
        for (uint32_t i = begin[l]; i < end[l]; i++) {
            const uint32_t m = pixels[i], c = m / rows;
            v += img[m];
            x += double(c < 128 ? c + 128 : c - 128) * img[m];
        }
        if (std::abs(mom[6 * l] - x) > 1e-9 * std::abs(x) || std::abs(mom[6 * l + 5] - v) > 1e-9 * std::abs(v)
            || ns[l] != int(end[l] - begin[l])) {
            std::printf("label %d: sums %g %g, should be %g %g\n", l, mom[6 * l], mom[6 * l + 5], x, v);
            bad++;
        }
    };
    run(SEG_BIG);
    check(0);
    std::printf("pixels read outside the image: %d\n", int(g_outside));
    bad += g_outside;
    for (uint32_t i = 0; i < large; i++) // sorted by the host
        pixels[small + i] = 400 + i;
    split[1] = small + large;
    run(~0u);
    check(0);
    check(1);
    bad += g_outside;

    // more labels than warps: a warp takes several, and small and large ones are summed in other ways; the sums of
    // each are those of its pixels in memory order (the ones from the split on first), to the last bit
    const int labels = 300;
    std::vector<uint32_t> b2, e2, sp2, px, li;
    for (int l = 0; l < labels; l++) {
        const uint32_t len = l % 7 == 0 ? 17 + l % 60 : 1 + l % 16;
        b2.push_back(uint32_t(px.size()));
        sp2.push_back(b2[l] + len / 3);
        for (uint32_t i = 0; i < len; i++)
            px.push_back((uint32_t(l) * 211u + i * 97u) % uint32_t(g_pixels));
        e2.push_back(uint32_t(px.size()));
        li.push_back(uint32_t((l * 7) % labels));
    }
    const uint32_t misc2[3] = { uint32_t(labels), 0, uint32_t(px.size()) }, nl2 = labels;
    std::vector<double> mom2(6 * labels, -1.0);
    std::vector<int> ns2(labels, -1);
    launch(Dim3 { 2, 1, 1 }, 32 * kSumWarps, [&] {
        k_label_sums<float>(FgSizes { misc2, uint32_t(labels), misc2[2] }, img.data(), rows, cols, px.data(), b2.data(),
            e2.data(), sp2.data(), li.data(), &nl2, SEG_BIG, mom2.data(), ns2.data());
    });
    for (int l = 0; l < labels; l++) {
        double s[6] = {};
        const uint32_t len = e2[l] - b2[l];
        for (uint32_t j = 0; j < len; j++) {
            const uint32_t m = px[seg_at(b2[l], sp2[l], e2[l], j)], c = m / rows, r = m % rows;
            const double x = double(c < 128 ? c + 128 : c - 128), y = double(r < 128 ? r + 128 : r - 128), v = img[m];
            const double xv = x * v, yv = y * v, terms[6] = { xv, yv, xv * x, yv * y, xv * y, v };
            for (int k = 0; k < 6; k++)
                s[k] += terms[k];
        }
        for (int k = 0; k < 6; k++)
            bad += s[k] != mom2[6 * l + k];
        bad += ns2[l] != int(len);
    }
    return bad ? 1 : 0;
}
