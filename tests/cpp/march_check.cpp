// The planner of segmentctscans_b200/csrc/march_plan.cuh against a plain restatement: every item by itself
// to the slot that is free first, the runs of columns found row by row.  Random masks (columns without
// rows, gaps, several volumes), tile shapes, slots and fixed segments; and a bound on its host time.
#include <chrono>
#include <cmath>
#include <cstdio>
#include <functional>
#include <queue>
#include <random>

#include "march_plan.cuh"

namespace {

struct Mask {
    std::vector<uint32_t> start, base;
    potts_mapping m{};

    Mask(int rows, int cols, int n_images, const std::function<RowRange(int)> &range)
        : start((size_t)cols), base((size_t)cols + 1)
    {
        m.rows = (uint32_t)rows, m.cols = (uint32_t)cols, m.n_images = (uint32_t)n_images;
        m.nstride = (uint32_t)(n_images + 3) / 4 * 4;
        m.col_begin = 0, m.col_end = (uint32_t)cols;
        for (int c = 0; c < cols; ++c) {
            const RowRange r = range(c);
            start[(size_t)c] = (uint32_t)r.first;
            base[(size_t)c + 1] = base[(size_t)c] + (uint32_t)(r.second - r.first) * m.nstride;
        }
        m.start_row = start.data();
        m.base = base.data();
    }
};

Mask cylinder(int n, int rows, int cols, double radius)
{
    return Mask(rows, cols, n, [=](int c) {
        const double d = c - (cols - 1) / 2.0, h = radius * radius - d * d;
        if (h <= 0) return RowRange{0, 0};
        const int lo = std::max(0, (int)std::ceil((rows - 1) / 2.0 - std::sqrt(h)));
        return RowRange{lo, std::min(rows, (int)std::floor((rows - 1) / 2.0 + std::sqrt(h)) + 1)};
    });
}

// Segment and time by the definition.
double plain(const std::vector<MarchVolume> &vols, int rows, int slices, int slots, int fixed, int *best)
{
    std::vector<std::pair<int, int>> runs;  // columns, tiles
    for (const MarchVolume &v : vols) {
        const potts_mapping &m = *v.map;
        const auto count = [&](int c) { return (int)((m.base[c + 1] - m.base[c]) / m.nstride); };
        int lo = INT32_MAX, hi = 0;
        for (int c = v.c_begin; c < v.c_end; ++c)
            if (count(c) > 0) {
                lo = std::min(lo, (int)m.start_row[c]);
                hi = std::max(hi, (int)m.start_row[c] + count(c));
            }
        for (int r0 = lo; r0 < hi; r0 += rows) {
            int len = 0;
            for (int c = v.c_begin; c <= v.c_end; ++c) {
                const bool in = c < v.c_end && count(c) > 0 && (int)m.start_row[c] < r0 + rows &&
                                (int)m.start_row[c] + count(c) > r0;
                if (!in && len > 0) runs.push_back({len, (v.ns + slices - 1) / slices});
                len = in ? len + 1 : 0;
            }
        }
    }
    double best_time = -1.0;
    for (int seg : kSegments) {
        if (fixed > 0) seg = fixed;
        std::vector<int> items;
        for (int k = 0; k < 70000; ++k) {
            const size_t before = items.size();
            for (const auto &r : runs)
                if (k * seg < r.first) items.insert(items.end(), (size_t)r.second, std::min(seg, r.first - k * seg));
            if (items.size() == before) break;
        }
        int64_t planes = 0;
        for (int len : items) planes += len + kItemPlanes;
        const bool many = (int64_t)items.size() >= (int64_t)kManyWaves * slots;
        double time = (double)planes / slots;
        if (!many && (best_time < 0.0 || time < best_time)) {
            std::priority_queue<int, std::vector<int>, std::greater<int>> ends;
            for (int i = 0; i < slots; ++i) ends.push(0);
            int last = 0;
            for (int len : items) {
                const int end = ends.top() + len + kItemPlanes;
                ends.pop();
                ends.push(end);
                last = std::max(last, end);
            }
            time = last;
        }
        if (best_time < 0.0 || time < best_time) {
            best_time = time;
            *best = seg;
        }
        if (fixed > 0 || (seg == kSegments[0] && many)) break;
    }
    return best_time;
}

}  // namespace

int main()
{
    std::mt19937 rng(3);
    const auto pick = [&](int lo, int hi) { return std::uniform_int_distribution<int>(lo, hi)(rng); };
    int wrong = 0, checks = 0;
    for (int rep = 0; rep < 120; ++rep) {
        std::vector<Mask> masks;
        const int n_vols = rep % 5 == 0 ? pick(2, 6) : 1;
        for (int i = 0; i < n_vols; ++i) {
            const int rows = pick(1, 180), cols = pick(1, 220), n = pick(1, 600);
            if (rep % 2)
                masks.push_back(cylinder(n, rows, cols, 0.47 * std::min(rows, cols)));
            else
                masks.emplace_back(rows, cols, n, [&](int) {
                    const int lo = pick(0, rows - 1);  // also of a column without rows
                    return RowRange{lo, pick(0, 5) == 0 ? lo : pick(lo, rows)};
                });
        }
        std::vector<MarchVolume> vols;
        for (Mask &k : masks) {
            k.m.start_row = k.start.data(), k.m.base = k.base.data();  // the vector may have moved them
            const int a = pick(0, (int)k.m.cols - 1);
            vols.push_back(rep % 3 ? MarchVolume{&k.m, (int)k.m.n_images, 0, (int)k.m.cols}
                                   : MarchVolume{&k.m, (int)k.m.n_images, a, pick(a, (int)k.m.cols)});
        }
        const int shapes[][2] = {{16, 64}, {8, 128}, {8, 64}, {4, 64}, {16, 128}};
        for (const auto &s : shapes) {
            const int slots = pick(0, 1) ? 148 * pick(1, 4) : pick(1, 40), fixed = pick(0, 2) ? 0 : pick(1, 64);
            int got = 64, want = 64;
            const double a = march_time(march_runs(vols, s[0]), s[1], slots, fixed, &got);
            const double b = plain(vols, s[0], s[1], slots, fixed, &want);
            wrong += a != b || got != want;
            ++checks;
        }
    }
    std::printf("plans: %d of %d differ\n", wrong, checks);
    // the choice of the gradient's segment for a 200^3 core: a part of its 60 us on the device
    const Mask core = cylinder(200, 200, 200, 94.0);
    double least = 1e9;
    for (int i = 0; i < 50; ++i) {
        const auto t0 = std::chrono::steady_clock::now();
        int seg = 0;
        march_time(march_runs({{&core.m, 200, 0, 200}}, 16), 128, 4 * 148, 0, &seg);
        least = std::min(least, std::chrono::duration<double, std::micro>(std::chrono::steady_clock::now() - t0).count());
    }
    std::printf("segment of a 200^3 core: %.1f us\n", least);
    return wrong != 0 || least > 60.0;
}
