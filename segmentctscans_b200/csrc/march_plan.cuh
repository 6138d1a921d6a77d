// Host-side planning of the column-march kernels: the runs of columns that a tile's rows lie in, and the
// column segment that the work items are cut into.  Plain C++ (tests/cpp/march_check.cpp compiles it).
// The whole choice runs in the first call on a mapping, so it must cost little beside an iteration: the
// columns' rows are divided out once per tile height, and the schedule is dealt out group by group.
// grad_magn of a 200^3 core in its first call on a mapping: 0.31 ms, 0.37 with a heap of slots and the
// divisions in every tile row (0.31 with a fixed segment).
#pragma once

#include <algorithm>
#include <cstdint>
#include <utility>
#include <vector>

#include "potts_b200.h"

namespace {

// The slices and columns that a column-march kernel runs over.
struct MarchVolume {
    const potts_mapping *map;
    int ns;
    int c_begin, c_end;
};

// Rows [first, second) of each of the columns [c_begin, c_end) (first = second: none).
using RowRange = std::pair<int, int>;

std::vector<RowRange> column_rows(const potts_mapping &m, int c_begin, int c_end)
{
    std::vector<RowRange> rows((size_t)std::max(c_end - c_begin, 0));
    for (int c = c_begin; c < c_end; ++c) {
        const uint32_t cnt = (m.base[c + 1] - m.base[c]) / m.nstride;
        if (cnt > 0) rows[(size_t)(c - c_begin)] = {(int)m.start_row[c], (int)(m.start_row[c] + cnt)};
    }
    return rows;
}

// First row and one past the last row of the columns ({0, 0}: no rows).
RowRange row_range(const std::vector<RowRange> &cols)
{
    RowRange all{INT32_MAX, 0};
    for (const RowRange &c : cols)
        if (c.first < c.second) all = {std::min(all.first, c.first), std::max(all.second, c.second)};
    return all.first < all.second ? all : RowRange{0, 0};
}

// Calls f(first, second) for each run of columns that hold rows of [r0, r0 + rows), counted from cols[0].
template <typename F>
void tile_runs(const std::vector<RowRange> &cols, int r0, int rows, F f)
{
    const int n = (int)cols.size();
    for (int c = 0, first = -1; c <= n; ++c) {
        // a column without rows has first = second = 0 and holds none of them
        const bool in = c < n && cols[(size_t)c].first < r0 + rows && cols[(size_t)c].second > r0;
        if (in && first < 0) first = c;
        if (!in && first >= 0) {
            f(first, c);
            first = -1;
        }
    }
}

// Column planes that a work item costs besides those of its columns: the plane
// before and after them, filling the load ring and the drain at its end.  With
// 4 the choice below was within 2 % (at most 9 %) of the best of 13 segment
// lengths on cores of 128^3 to 203 x 301 x 287 voxels, three shapes and both arithmetics.
constexpr int kItemPlanes = 4;
constexpr int kSegments[] = {64, 48, 40, 32, 24, 20, 16, 12, 10, 8, 6};

// The runs of all tile rows of some volumes: columns, and the slices of the volume.
struct MarchRun {
    int len, ns;
};

std::vector<MarchRun> march_runs(const std::vector<MarchVolume> &vols, int rows)
{
    std::vector<MarchRun> runs;
    for (const MarchVolume &v : vols) {
        const std::vector<RowRange> cols = column_rows(*v.map, v.c_begin, v.c_end);
        const RowRange all = row_range(cols);
        for (int r0 = all.first; r0 < all.second; r0 += rows)
            tile_runs(cols, r0, rows, [&](int first, int second) { runs.push_back({second - first, v.ns}); });
    }
    return runs;
}

// Expected time of the volumes' work items for tiles of `slices` slices and the rows of `runs` (in planes of
// one tile), and the segment length that gives it (`segment` > 0: that one).  A
// block runs one item and `slots` blocks run at a time, so a volume of few tiles
// leaves multiprocessors idle, or its last wave nearly empty, with long segments,
// and pays kItemPlanes too often with short ones: 128^3 (radius 60, fast, 8 x
// 128 tiles) takes 171 us per iteration with segments of 64 columns (30 items), 52
// with 10 and 57 with 4.  The items go to the first free slot in order, as the
// hardware hands out blocks; with at least kManyWaves items per slot their mean decides.
constexpr int kManyWaves = 12;
double march_time(const std::vector<MarchRun> &runs, int slices, int slots, int segment, int *best)
{
    const auto tiles = [&](const MarchRun &r) { return (r.ns + slices - 1) / slices; };
    double best_time = -1.0;
    std::vector<int> free_at;  // slots that become free after so many planes
    for (int seg : kSegments) {
        if (segment > 0) seg = segment;
        int64_t items = 0, planes = 0;
        int longest = 0;  // segments of the longest run
        for (const MarchRun &r : runs) {
            const int n = (r.len + seg - 1) / seg;
            items += (int64_t)n * tiles(r);
            planes += (int64_t)(r.len + n * kItemPlanes) * tiles(r);
            longest = std::max(longest, n);
        }
        double time = (double)planes / slots;
        if (items < (int64_t)kManyWaves * slots && (best_time < 0.0 || time < best_time)) {
            free_at.assign((size_t)(planes / slots + 2 * (seg + kItemPlanes) + 2), 0);
            free_at[0] = slots;
            int now = 0, end = 0;
            for (int k = 0; k < longest; ++k)
                for (const MarchRun &r : runs) {
                    if (k * seg >= r.len) continue;
                    const int cost = std::min(seg, r.len - k * seg) + kItemPlanes;
                    for (int left = tiles(r); left > 0;) {
                        while (free_at[(size_t)now] == 0) ++now;
                        const int n = std::min(left, free_at[(size_t)now]);
                        free_at[(size_t)now] -= n;
                        free_at[(size_t)(now + cost)] += n;
                        left -= n;
                        end = std::max(end, now + cost);
                    }
                }
            time = (double)end;
        }
        if (best_time < 0.0 || time < best_time) {
            best_time = time;
            *best = seg;
        }
        // many items with the longest segments: shorter ones only add planes
        if (segment > 0 || (seg == kSegments[0] && items >= (int64_t)kManyWaves * slots)) break;
    }
    return best_time;
}

}  // namespace
