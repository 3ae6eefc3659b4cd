// partition.h -- neighbouring cavities of a batch put into groups that are stepped
// together (host C++ only: tests/native/partition_check.cpp compiles it alone).
#pragma once

#include <algorithm>
#include <cstddef>
#include <vector>

namespace cav {

// What a step of a group costs, in bytes moved at the L2's rate: its state, each
// byte dearer once the state no longer stays in the L2 from step to step, and a
// launch with its start and last wave.  Fitted to the 64-cavity sweep (2.29 M
// nodes: 340 MB in FP32, 175 MB in 16 bits) on a B200 (L2 of 132.6 MB), us per
// lattice step against the groups' size in MB:
//   FP32  (k_batch_np)      340: 61.9   85: 52.5   68: 46.3   57: 46.0   42: 47.4
//   f16sr (k_batch_x, r 2)  175: 48.6   87: 43.8   58: 40.0   44: 41.5   35: 42.6
// (0.12 us per MB up to 56 MB, 0.126 at 68, 0.146 at 85, 0.18 where nothing stays;
// 0.7 - 1.3 us a launch).  The quadratic also evens the groups out.
constexpr double GROUP_LAUNCH = 8e6, GROUP_FITS = 0.42, GROUP_RISE = 1.1, GROUP_MISS = 0.46;

inline double group_cost(double bytes, double l2) {
    const double over = std::max((bytes - GROUP_FITS * l2) / (l2 - GROUP_FITS * l2), 0.0);
    return GROUP_LAUNCH + bytes * (1.0 + std::min(GROUP_RISE * over * over, GROUP_MISS));
}

// First cavity of every group, and their number at the end: the cheapest cut of
// the list (by dynamic programming over its prefixes) among those whose groups
// are single cavities or hold at most four times the L2.
inline std::vector<int> partition_groups(const std::vector<size_t>& bytes, size_t l2) {
    const int n = int(bytes.size());
    std::vector<double> best(n + 1, 0.0);
    std::vector<int> from(n + 1, 0);
    for (int j = 1; j <= n; ++j) {
        double sum = 0.0;
        for (int i = j - 1; i >= 0; --i) {  // a group [i, j)
            sum += double(bytes[i]);
            if (i < j - 1 && sum > 4.0 * double(l2)) break;
            const double c = best[i] + group_cost(sum, double(l2));
            if (i == j - 1 || c < best[j]) {
                best[j] = c;
                from[j] = i;
            }
        }
    }
    std::vector<int> first{n};
    for (int j = n; j > 0; j = from[j]) first.push_back(from[j]);
    std::reverse(first.begin(), first.end());
    return first;
}

}  // namespace cav
